// Fused gather-matmul-scatter on the 5th-generation tensor cores (tcgen05 + tensor
// memory), fp16 in / fp32 accumulate, output stationary, persistent and warp-specialised.  Two
// kernels share lists, shares and options: k_conv_deep (one CTA per SM, rows by TMA gathers) takes
// the layers whose input width is a multiple of 32, k_conv_umma, described first, all others, halo
// pushes and narrow layers on large maps; the rule stands in conv_umma_impl.
//
// The kernel reads the map as TILE LISTS (built once per kernel map by pce_build_tile_lists):
// output rows are taken in sorted order (pce_csr_sort_rows) in tiles of 128 or 256; for every
// tile the offsets that at least one of its rows has are listed (`stage_kp`), each with the
// input row to fetch per tile row (`stage_nbr`, -1 = this row lacks the offset).  A stage is one
// (tile, offset); offsets nobody in the tile has cost nothing (the indicator).  Lists built with
// the identity stage end every tile with a stage in which each row names itself: there a second
// operand (a residual block's shortcut) joins the accumulation.
//
// One CTA owns a contiguous range of tiles holding about 1/gridDim of the work and
// streams through that range's stages.  Threads (SUB = 128-row sub-tiles per tile):
//   4*SUB producer warps, one thread per tile row: per stage and 64-channel K block they
//              gather the input rows with 16-byte cp.async (4 rows per warp instruction,
//              full 128-byte lines, zero-fill for -1) into a 128-byte-swizzled K-major tile and
//              attach the stage's barrier to the copies (cp.async.mbarrier.arrive.noinc): the
//              barrier fires when the data has landed, the thread does not wait for it.
//              Thread 0 also stages the pre-packed weight block with one bulk async copy
//              (cp.async.bulk, the TMA engine).  Stage indices are read four stages ahead
//              (coalesced reads) into registers that are never moved, so the loads stay in
//              flight until the stage that uses them.
//              (tile::gather4 costs its warp 43 ns an operation: too slow from a few warps, and
//              what k_conv_deep below spreads over sixteen.)
//   one MMA warp: one lane issues tcgen05.mma (M=128, N=C_out, K=16; one per sub-tile on the
//              same weight descriptor) and commits to mbarriers.
//   4 epilogue warps: tcgen05.ld the finished accumulator, apply
//              act(acc*scale + shift + residual), convert to fp16, store each row once (and, in
//              the PUSH variant, boundary rows a second time into a neighbouring GPU's halo).
// Rings: kStages smem stages (afull / bfull / empty mbarriers) that run on across tile
// boundaries, and one or two accumulator sets in tensor memory (accfull / accempty); with two,
// the gather of tile i+1, the MMAs of tile i and the stores of tile i-1 overlap.
// No atomics, no intermediate buffer in HBM, bit-identical run to run.
//
// Every mbarrier wait is bounded (~1 s): when one expires the CTA raises an abort flag,
// records PCE_ERR_TIMEOUT in the library's device status word, drains its own copies,
// frees its tensor memory and returns.
//
// Replaces fetch_on_demand_gemm_fp16_tc4_async and the cuBLAS centre GEMM of the
// reference (ref: backend/spconv.cuh:1567-1730, backend/spconv.cu:273-298,338).
#include <cuda.h>

#include "common.cuh"

namespace pce {

__device__ int g_umma_status = 0;
// Where the first bounded wait of a launch gave up: {code, CTA, item, extra}; code = role | sub-tile << 4 |
// tile-in-CTA << 8 with role 1 producer/row slot free, 2 loader/weight slot free, 3 MMA/weights landed,
// 4 MMA/accumulator drained, 5 MMA/rows landed, 6 MMA/accumulator drained (nothing written), 7 epilogue/
// accumulator complete (k_conv_umma_mt), 9 any wait of k_conv_umma.
__device__ int g_umma_where[4] = {0, 0, 0, 0};

namespace umma {

constexpr int kTileM = 128;
constexpr int kMaxStages = 4;
constexpr int kABytes = kTileM * 128;  // one A stage: 128 rows x 64 fp16
constexpr long long kWaitCycles = 2000000000ll;  // ~1 s at 2 GHz

struct Epi {
  const float* scale;
  const float* shift;
  const __half* residual;
  int act;
  float slope;
  // halo push: output row r is also stored to push_base[s] + push_slot[s][r] * cout (slot >= 0), memory
  // of a neighbouring GPU mapped into this process (plain peer stores over NVLink)
  const int* push_slot[2];
  __half* push_base[2];
  // row pitch of the input and the output features in elements (the channel count when dense): a layer
  // may read and write a column range of a wider row-major matrix
  int ld_in;
  int ld_out;
  // parts > 1: a cluster of `parts` CTAs shares every tile (CTA b: tile b / parts, part b % parts of its stage list).
  // Each leaves its fp32 sums in its own shared memory, and finishes its part of the tile's rows from all of them.
  int parts;
  float* partial;
  // streamk: every CTA takes an equal share of the layer's STAGES (CTA b: stages S*b/G .. S*(b+1)/G of the
  // concatenated tile lists), whatever tiles they fall in.  A tile that lies in one CTA's share is finished by
  // it; a tile cut between CTAs leaves raw fp32 sums in partial[((cta*2 + slot)*128 + row-in-tile)*cout + c]
  // (slot 0: the CTA's first tile, 1: its last) and k_sum_cut_tiles finishes it.
  int streamk;
};

struct Lists {
  const int* order;      // [n_out] processing order of the output rows, or nullptr (natural)
  const int* tile_ptr;   // [n_tiles+1] first stage of every tile, or nullptr (dense product)
  const int* stage_kp;   // [stages] offset of every stage
  const int* stage_nbr;  // [stages][tile rows] input row per tile row, -1 absent
  int identity;          // every tile's last stage is the identity stage (stage_kp = -1)
  const __half* wtail;   // the weights' 32-channel image, for the last K block of a width that is an odd multiple of 32
  const __half* wslots;  // SLOTS > 1: weights as [kv][cout][cin] (one 16-byte chunk row per output channel)
  int settled;           // the lists were complete before the previous kernel of the stream was launched
  int entries;           // k_conv_deep: offsets per listed stage (1 or 2), each a ring stage of its own there
  int tall;              // k_conv_deep: the lists' tiles are 256 rows, two of the kernel's
};

// Second operand: out[row] += in2[row] @ w2, joined to the accumulation at the identity stage.
// The residual of a block (w2 = identity matrix) and its 1x1x1 shortcut convolution take this path.
struct Second {
  const __half* in2;  // [n_out][cin2], nullptr: none
  const __half* w2;   // packed like the weights of one offset: kblocks2 images of cout x 128 B
  const __half* wtail;  // as Lists::wtail
  int cin2;
};

struct SharedCtl {
  unsigned long long afull[kMaxStages];
  unsigned long long bfull[kMaxStages];
  unsigned long long empty[kMaxStages];
  unsigned long long accfull[2];
  unsigned long long accempty[2];
  uint32_t tmem_base;
  int range[2];  // this CTA's tiles [range[0], range[1])
  volatile int abort_flag;
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("{\n\t.reg .b64 st;\n\tmbarrier.arrive.shared::cta.b64 st, [%0];\n\t}" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("{\n\t.reg .b64 st;\n\tmbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1;\n\t}" ::"r"(bar),
               "r"(bytes)
               : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.b32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}

// Bounded wait: false when the abort flag is up or the deadline passed.
template <class Ctl>
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, Ctl* ctl, int where = 9, int item = 0) {
  if (mbar_try_wait(bar, parity)) return true;
  const long long t0 = clock64();
  int spins = 0;
  while (!mbar_try_wait(bar, parity)) {
    if (((++spins) & 255) == 0) {
      if (ctl->abort_flag) return false;
      if (clock64() - t0 > kWaitCycles) {
        ctl->abort_flag = 1;
        atomicMax(&g_umma_status, PCE_ERR_TIMEOUT);
        if (atomicCAS(&g_umma_where[0], 0, where) == 0) {
          g_umma_where[1] = static_cast<int>(blockIdx.x);
          g_umma_where[2] = item;
          g_umma_where[3] = static_cast<int>(parity);
        }
        return false;
      }
    }
  }
  return true;
}

// One lane of a fully active warp.  Tensor-core, commit and bulk-copy instructions want uniform operands and a single
// issuing thread, which the compiler can prove behind `elect.sync` but not behind `if (lane == 0)`: there a 64-channel
// stage's four products and commit took about 1000 cycles to ISSUE (their execution 130 to 200), more than anything
// else in the kernel; elected, and with the four steps unrolled, about 500.  Whole layers: 96->96 on 240 k rows
// 50 -> 46 us, 128->128 on 137 k rows 50 -> 44 us, 256->256 on 58 k rows 83 -> 74 us.
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xFFFFFFFF;\n\tselp.b32 %0, 1, 0, p;\n\t}" : "=r"(p));
  return p != 0;
}

__device__ __forceinline__ void bulk_copy_g2s(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, uint32_t src_bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(src_bytes) : "memory");
}
// Makes the mbarrier receive one (already counted) arrival once every cp.async this thread has
// issued so far has landed: the thread itself does not wait.
__device__ __forceinline__ void cp_async_arrive_noinc(uint32_t bar) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void tc_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

// D[tmem] (+)= A[smem desc] * B[smem desc]; fp16 operands, fp32 accumulate.
__device__ __forceinline__ void tc_mma_f16(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc,
                                           uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
      "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
      : "memory");
}

// The same with the descriptors' halves apart.
__device__ __forceinline__ void tc_mma_f16_lohi(uint32_t tmem_d, uint32_t a_lo, uint32_t a_hi, uint32_t b_lo, uint32_t b_hi, uint32_t idesc,
                                                uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 a, b;\n\tsetp.ne.b32 p, %6, 0;\n\tmov.b64 a, {%1, %2};\n\tmov.b64 b, {%3, %4};\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %5, p;\n\t}" ::"r"(tmem_d),
      "r"(a_lo), "r"(a_hi), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(accumulate)
      : "memory");
}

// K-major, 128-byte swizzle: rows of 128 B, 8-row groups 1024 B apart, descriptor version 1.
__device__ __forceinline__ uint64_t make_desc(uint32_t smem_addr) {
  const uint32_t lo = ((smem_addr >> 4) & 0x3FFFu) | (1u << 16);
  const uint32_t hi = (1024u >> 4) | (1u << 14) | (2u << 29);
  return (static_cast<uint64_t>(hi) << 32) | lo;
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, "
      "[%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, "
      "%18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
        "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]),
        "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
        "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ uint32_t pack_half2(uint32_t lo, uint32_t hi) {
  const __half2 h = __floats2half2_rn(__uint_as_float(lo), __uint_as_float(hi));
  return *reinterpret_cast<const uint32_t*>(&h);
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// 32 bytes of a row in ONE store (256-bit vector access): half the store instructions, and half the requests to
// the load/store unit, of two 16-byte stores; `p` must be 32-byte aligned.
__device__ __forceinline__ void store32(void* p, const uint4& a, const uint4& b) {
  asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w),
               "r"(b.x), "r"(b.y), "r"(b.z), "r"(b.w)
               : "memory");
}

__device__ __forceinline__ void load32(const void* p, uint4& a, uint4& b) {
  asm volatile("ld.global.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(a.x), "=r"(a.y), "=r"(a.z), "=r"(a.w), "=r"(b.x), "=r"(b.y), "=r"(b.z), "=r"(b.w)
               : "l"(p)
               : "memory");
}

__device__ __forceinline__ float act_apply(float v, int act, float slope) {
  if (act == PCE_ACT_RELU) return v > 0.f ? v : 0.f;
  if (act == PCE_ACT_LEAKY) return v > 0.f ? v : v * slope;
  return v;
}

// Weights [kv][cin][cout] fp16 -> per (kp, k-block) shared-memory images of cout rows x 128 B
// (64 K elements, zero padded), 16-byte chunks XOR-swizzled with the row index.
// kb_size = 32: images of cout rows x 64 B (32 K elements), 64-byte swizzle (chunk ^ ((row >> 1) & 3)).
__global__ void k_pack_weights(const __half* __restrict__ w, int kv, int cin, int cout, int kblocks,
                               __half* __restrict__ packed, int kb_size) {
  if (kb_size == 32) {
    const long long total32 = static_cast<long long>(kv) * kblocks * cout * 32;
    for (long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i < total32;
         i += static_cast<long long>(gridDim.x) * blockDim.x) {
      const int kk = static_cast<int>(i % 32);
      long long t = i / 32;
      const int co = static_cast<int>(t % cout);
      t /= cout;
      const int kb = static_cast<int>(t % kblocks);
      const int kp = static_cast<int>(t / kblocks);
      const int ci = kb * 32 + kk;
      __half v = __float2half(0.f);
      if (ci < cin) v = w[(static_cast<size_t>(kp) * cin + ci) * cout + co];
      const int chunk = kk >> 3, within = kk & 7;
      const size_t img = (static_cast<size_t>(kp) * kblocks + kb) * cout * 32;
      packed[img + static_cast<size_t>(co) * 32 + ((chunk ^ ((co >> 1) & 3)) << 3) + within] = v;
    }
    return;
  }
  const long long total = static_cast<long long>(kv) * kblocks * cout * 64;
  for (long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i < total;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int kk = static_cast<int>(i % 64);
    long long t = i / 64;
    const int co = static_cast<int>(t % cout);
    t /= cout;
    const int kb = static_cast<int>(t % kblocks);
    const int kp = static_cast<int>(t / kblocks);
    const int ci = kb * 64 + kk;
    __half v = __float2half(0.f);
    if (ci < cin) v = w[(static_cast<size_t>(kp) * cin + ci) * cout + co];
    const int chunk = kk >> 3, within = kk & 7;
    const size_t img = (static_cast<size_t>(kp) * kblocks + kb) * cout * 64;
    packed[img + static_cast<size_t>(co) * 64 + ((chunk ^ (co & 7)) << 3) + within] = v;
  }
}

// Weights [kv][cin][cout] -> [kv][cout][cin]: per offset and output channel the cin input-channel values in a row.
__global__ void k_pack_weight_slots(const __half* __restrict__ w, int kv, int cin, int cout, __half* __restrict__ out) {
  const long long total = static_cast<long long>(kv) * cout * cin;
  for (long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i < total;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int ci = static_cast<int>(i % cin);
    const long long t = i / cin;
    const int co = static_cast<int>(t % cout);
    const int kp = static_cast<int>(t / cout);
    out[i] = w[(static_cast<size_t>(kp) * cin + ci) * cout + co];
  }
}

// Work of tiles [0, t): `unit` per stage, and one per tile for its fixed cost (the epilogue).  A listed offset of up to 64
// channels costs about what the tile itself does, a wider one twice that (64->64 on 1.5 M rows 118 us with 1:1, 123 with
// 2:1; 128->128 on 200 k rows 53 with 1:1, 51 with 2:1).
__device__ __forceinline__ long long cost_before(const int* tile_ptr, int t, int unit, int fixed = 1) {
  return static_cast<long long>(unit) * (tile_ptr ? static_cast<long long>(__ldg(tile_ptr + t)) : static_cast<long long>(t)) +
         static_cast<long long>(fixed) * t;
}

// The tile that begins nearest to the point where the work reaches `target`: a share then misses its due by at most half
// a tile at each end.  (Cut at the first tile behind that point it was a whole tile at one end, and tiles hold 1 to 27
// stages where a share holds about 15.)  cost_before is strictly increasing.  Found by a whole warp: 32 probes per round, so a list of n tiles takes log32(n) dependent loads instead of the
// log2(n) of a binary search (about 20 L2 round trips per CTA for both ends of its range, a fixed
// 15 us that was a tenth of the large layers and a third of the small ones).
__device__ __forceinline__ int warp_tile_at_cost(const int* tile_ptr, int n_tiles, long long target, int unit, int lane, int fixed = 1) {
  int lo = 0, hi = n_tiles;  // the answer lies in [lo, hi]
  while (lo < hi) {
    const int step = (hi - lo + 31) / 32;
    const int p = min(lo + (lane + 1) * step - 1, hi - 1);
    const unsigned m = __ballot_sync(0xFFFFFFFFu, cost_before(tile_ptr, p, unit, fixed) >= target);
    if (m == 0) {  // no tile in [lo, hi) reaches the target
      lo = hi;
      break;
    }
    const int f = __ffs(m) - 1;
    const int hit = min(lo + (f + 1) * step - 1, hi - 1);
    lo = f == 0 ? lo : min(lo + f * step - 1, hi - 1) + 1;
    hi = hit;
  }
  if (lo > 0 && target - cost_before(tile_ptr, lo - 1, unit, fixed) < cost_before(tile_ptr, lo, unit, fixed) - target) --lo;
  return lo;
}

__device__ __forceinline__ int first_stage(const int* tile_ptr, int t) { return tile_ptr ? __ldg(tile_ptr + t) : t; }

// First tile t in [0, n_tiles) with tile_ptr[t + 1] > s (the tile that holds stage s), by a whole warp;
// n_tiles when there is none.
__device__ __forceinline__ int warp_tile_of_stage(const int* tile_ptr, int n_tiles, int s, int lane) {
  int lo = 0, hi = n_tiles;
  while (lo < hi) {
    const int step = (hi - lo + 31) / 32;
    const int p = min(lo + (lane + 1) * step - 1, hi - 1);
    const unsigned m = __ballot_sync(0xFFFFFFFFu, __ldg(tile_ptr + p + 1) > s);
    if (m == 0) return hi;
    const int f = __ffs(m) - 1;
    const int hit = min(lo + (f + 1) * step - 1, hi - 1);
    lo = f == 0 ? lo : min(lo + f * step - 1, hi - 1) + 1;
    hi = hit;
  }
  return lo;
}

// Share of CTA b of G in S stages: [S*b/G, S*(b+1)/G).
__host__ __device__ __forceinline__ int share_begin(long long total, int b, int g) {
  return static_cast<int>(total * b / g);
}

__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}
// 16 bytes at this address of the shared memory of CTA `rank` of the cluster.
__device__ __forceinline__ float4 cluster_ld4(uint32_t addr, int rank) {
  uint32_t there;
  float4 v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(there) : "r"(addr), "r"(rank));
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"(there)
               : "memory");
  return v;
}

// The last steps for eight channels of a row whose sums (scaled and shifted) are complete: residual, activation, store.
__device__ __forceinline__ void finish8(float (&v)[8], int row, int c0, int cout, __half* out, const Epi& ep) {
  if (ep.residual) {
    const uint4 r = *reinterpret_cast<const uint4*>(ep.residual + static_cast<size_t>(row) * cout + c0);
    const __half2* h = reinterpret_cast<const __half2*>(&r);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const float2 f = __half22float2(h[q]);
      v[2 * q] += f.x;
      v[2 * q + 1] += f.y;
    }
  }
  uint4 o;
  __half2* po = reinterpret_cast<__half2*>(&o);
#pragma unroll
  for (int q = 0; q < 4; ++q)
    po[q] = __floats2half2_rn(act_apply(v[2 * q], ep.act, ep.slope), act_apply(v[2 * q + 1], ep.act, ep.slope));
  *reinterpret_cast<uint4*>(out + static_cast<size_t>(row) * ep.ld_out + c0) = o;
}

// kStages = depth of the smem stage ring.  SUB = 128-row sub-tiles per tile (1 or 2): a tile of 128*SUB output rows
// has SUB accumulators and every staged weight block feeds SUB MMAs, which halves the weight
// traffic per row for SUB = 2.  Threads: 4*SUB producer warps, the MMA warp, 4 epilogue warps.
// SLOTS = offsets per stage (1, 2, 4): with 32 or 16 input channels an offset fills half or a quarter
// of the 64-channel K block, so SLOTS offsets of a tile share one ring stage: every row gathers one
// neighbour per slot into its part of the 128-byte row, and the producers assemble the stage's weight
// block from the per-offset images with cp.async (covered by the same barrier as the rows).
// K blocks are 64 channels, the last one padded in the weights.
template <int kStages, int SUB, bool PUSH, int SLOTS>
__global__ void __launch_bounds__(32 * (4 * SUB + 5), SUB == 1 ? 3 : 2)
    k_conv_umma(const __half* __restrict__ in, const __half* __restrict__ wpacked, Lists ls, Second sec, int n_out, int cin,
                int cout, __half* __restrict__ out, Epi ep, int tmem_cols, int nacc) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_addr = smem_u32(smem_raw);
  const uint32_t pad = ((raw_addr + 1023u) & ~1023u) - raw_addr;
  uint8_t* tiles = smem_raw + pad;  // 1024-byte aligned
  const uint32_t tiles_addr = raw_addr + pad;
  constexpr int KB = 64;                       // channels per K block
  constexpr int kRowBytes = KB * 2;            // one operand row of a stage
  const int b_bytes = cout * kRowBytes;
  constexpr int kRows = kTileM * SUB;          // output rows per tile
  constexpr int kAStage = kTileM * kRowBytes * SUB;  // gathered rows of one stage
  constexpr int kMmaWarp = 4 * SUB;
  const int stage_bytes = kAStage + b_bytes;   // both multiples of 1024
  SharedCtl* ctl = reinterpret_cast<SharedCtl*>(tiles + kStages * stage_bytes);
  // per-channel scale [cout] and shift [cout] of the epilogue (1 and 0 where absent), staged once per CTA: every
  // epilogue thread needs all of them for every tile, and read through the global path they cost the epilogue
  // eight 16-byte loads per 16-channel piece (96->96 on 486 k rows: 104 us without scale/shift, 146 us with)
  float* affine = reinterpret_cast<float*>(ctl + 1);
  static_assert(sizeof(SharedCtl) % 16 == 0, "the staged scale/shift are read as float4");

  const int tid = threadIdx.x;
  const int warp = tid >> 5;
  const int lane = tid & 31;
  const int kblocks = (cin + KB - 1) / KB;
  const int kblocks2 = sec.in2 ? (sec.cin2 + KB - 1) / KB : 0;  // ring stages of the identity stage
  const int n_tiles = (n_out + kRows - 1) / kRows;
  if (tid == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(smem_u32(&ctl->afull[s]), kRows);
      mbar_init(smem_u32(&ctl->bfull[s]), 1);
      mbar_init(smem_u32(&ctl->empty[s]), 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(smem_u32(&ctl->accfull[s]), 1);
      mbar_init(smem_u32(&ctl->accempty[s]), 128);
    }
    ctl->abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp > kMmaWarp && (ep.scale || ep.shift)) {  // (constants of the layer, not outputs of the previous kernel)
    for (int c = tid - 32 * (kMmaWarp + 1); c < cout; c += 128) {
      affine[c] = ep.scale ? __ldg(ep.scale + c) : 1.f;
      affine[cout + c] = ep.shift ? __ldg(ep.shift + c) : 0.f;
    }
  }
  if (warp == kMmaWarp) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&ctl->tmem_base)),
                 "r"(static_cast<uint32_t>(tmem_cols))
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  // Launched with programmatic stream serialisation: everything above ran while the kernel before
  // this one in the stream was still finishing; the features and the output buffer may not be touched
  // before that kernel has completed and its writes are visible.  The tile lists may, when they are
  // older than that kernel (ls.settled): the search for this CTA's tiles and the first index loads
  // then overlap its tail as well.
  if (!ls.settled) asm volatile("griddepcontrol.wait;" ::: "memory");
  const int parts = ep.parts > 1 ? ep.parts : 1;
  const bool streamk = ep.streamk != 0;
  int sk_begin = 0, sk_end = 0;  // this CTA's share of the stages (streamk)
  if (streamk) {
    const long long total = __ldg(ls.tile_ptr + n_tiles);
    sk_begin = share_begin(total, static_cast<int>(blockIdx.x), static_cast<int>(gridDim.x));
    sk_end = share_begin(total, static_cast<int>(blockIdx.x) + 1, static_cast<int>(gridDim.x));
    if (warp < 2) {
      int t = 0;
      if (sk_end > sk_begin) t = warp_tile_of_stage(ls.tile_ptr, n_tiles, warp == 0 ? sk_begin : sk_end - 1, lane) + warp;
      if (lane == 0) ctl->range[warp] = t;
    }
  } else if (parts > 1) {
    // split tiles: this CTA owns ONE tile and one part of its stage list
    if (tid == 0) {
      ctl->range[0] = static_cast<int>(blockIdx.x) / parts;
      ctl->range[1] = static_cast<int>(blockIdx.x) / parts + 1;
    }
  } else if (warp < 2) {
    // this CTA's contiguous share of the tiles, balanced by work: warp 0 finds its first tile,
    // warp 1 the next CTA's first tile
    const int unit = kblocks > 1 ? 2 : 1;
    const long long total = cost_before(ls.tile_ptr, n_tiles, unit);
    const unsigned b = blockIdx.x + warp;
    const int t = b >= gridDim.x ? n_tiles : warp_tile_at_cost(ls.tile_ptr, n_tiles, total * b / gridDim.x, unit, lane);
    if (lane == 0) ctl->range[warp] = t;
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = ctl->tmem_base;

  const int t0 = ctl->range[0], t1 = ctl->range[1];
  // stage range of a tile (its stages [sa, sb)) that this CTA works on: the whole tile, or its part
  auto stage_range = [&](int& sa, int& sb) {
    if (streamk) {
      sa = max(sa, sk_begin);
      sb = min(sb, sk_end);
    } else if (parts > 1) {
      const int n = sb - sa, part = static_cast<int>(blockIdx.x) % parts;
      const int a = sa + static_cast<int>(static_cast<long long>(n) * part / parts);
      sb = sa + static_cast<int>(static_cast<long long>(n) * (part + 1) / parts);
      sa = a;
    }
  };
  // The tiles' bounds, read a tile ahead: between two tiles the accumulator's hand-over is all there is to wait for.
  // main: ring stages of the listed offsets (of this CTA's part); ident: with the identity stage, which is the tile's
  // last and counts with the second operand's K blocks (none without one); cut: stream-K, only a piece of the tile.
  struct Work {
    int main, ident;
    bool cut;
  };
  int bound0 = 0, bound1 = 0, bound2 = 0;
  auto first_bounds = [&]() {
    bound1 = first_stage(ls.tile_ptr, t0);
    bound2 = t0 < t1 ? first_stage(ls.tile_ptr, t0 + 1) : bound1;
  };
  auto next_work = [&](int t) {
    bound0 = bound1;
    bound1 = bound2;
    if (t + 1 < t1) bound2 = first_stage(ls.tile_ptr, t + 2);
    int sa = bound0, sb = bound1;
    stage_range(sa, sb);
    Work w;
    w.ident = (ls.identity && sb > sa && sb == bound1) ? 1 : 0;
    w.main = (sb - sa - w.ident) * kblocks;
    w.cut = streamk && (sa > bound0 || sb < bound1);
    return w;
  };

  bool part_any = false;  // epilogue warps of a split tile: this CTA's part has products
  if (warp < kMmaWarp) {
    // =========================== producers ===========================
    int g0 = first_stage(ls.tile_ptr, t0), g1 = first_stage(ls.tile_ptr, t1);
    if (parts > 1) stage_range(g0, g1);
    if (streamk) {
      g0 = sk_begin;
      g1 = sk_end;
    }
    constexpr int kCpr = KB / 8;                // 16-byte chunks per operand row (8 or 4)
    constexpr int kRowsPerInstr = 32 / kCpr;    // rows one warp instruction covers (4 or 8)
    const int rsub = lane / kCpr;   // row inside the group of rows of one instruction
    const int chunk = lane % kCpr;  // 16-byte chunk inside the row
    int j = 0;  // smem stages issued so far (continuous over tiles)
    bool ok = true;
    // destination of this thread's copy q inside a stage: row q * kRowsPerInstr + rsub of the warp's 32, chunk
    // swizzled with the row; the swizzle term takes two values (q even / odd), everything else is q * constant
    const int sw_even = chunk ^ rsub;
    const int sw_odd = chunk ^ (rsub + 4);
    const uint32_t dst_even = (warp * 32 + rsub) * kRowBytes + (sw_even << 4);
    const uint32_t dst_odd = (warp * 32 + rsub) * kRowBytes + (sw_odd << 4);
    if constexpr (SLOTS == 1) {
    auto load_stage = [&](int g, int& nid, int& kp) {
      nid = -1;
      kp = 0;
      if (g < g1) {
        if (ls.tile_ptr) {
          nid = __ldg(ls.stage_nbr + static_cast<size_t>(g) * kRows + tid);
          kp = __ldg(ls.stage_kp + g);
          if (kp >= 0) kp &= 255;  // bits 8.. hold the sub-tile presence mask (read by k_conv_umma_mt)
        } else {  // dense product: stage g is tile g, every row fetches itself at offset 0
          const int row = g * kRows + tid;
          nid = row < n_out ? row : -1;
        }
      }
    };
    auto run_stage = [&](int nid, int kp) {
      const bool second = kp < 0;  // the identity stage
      const char* src_base = reinterpret_cast<const char*>(second ? sec.in2 : in) + chunk * 16;
      const int width = second ? sec.cin2 : cin;
      const int pitch_bytes = (second ? sec.cin2 : ep.ld_in) * 2;
      const int nkb = second ? kblocks2 : kblocks;  // 0: listed, but this launch has no second operand
      // the rows this thread fetches in this stage (the same for every K block)
      int rows[kCpr];
#pragma unroll
      for (int q = 0; q < kCpr; ++q) rows[q] = __shfl_sync(0xFFFFFFFFu, nid, q * kRowsPerInstr + rsub);
      for (int kb = 0; kb < nkb; ++kb, ++j) {
        const int s = j % kStages;
        const int n = j / kStages;
        if (n > 0) ok = mbar_wait(smem_u32(&ctl->empty[s]), (n - 1) & 1, ctl);
        ok = __all_sync(0xFFFFFFFFu, ok);  // keep the warp convergent
        if (!ok) return;
        const uint32_t a_addr = tiles_addr + s * stage_bytes;
        if (warp == 0 && elect_one()) {
          const uint32_t bbar = smem_u32(&ctl->bfull[s]);
          mbar_arrive_expect_tx(bbar, static_cast<uint32_t>(b_bytes));
          const __half* wsrc = second ? sec.w2 + static_cast<size_t>(kb) * cout * KB
                                      : wpacked + (static_cast<size_t>(kb) + static_cast<size_t>(kp) * kblocks) * cout * KB;
          bulk_copy_g2s(a_addr + kAStage, wsrc, static_cast<uint32_t>(b_bytes), bbar);
        }
        if (chunk < min(kCpr, (width - kb * KB) >> 3)) {
          const char* src_kb = src_base + kb * (KB * 2);
#pragma unroll
          for (int q = 0; q < kCpr; ++q) {
            const int row = rows[q];
            const uint32_t dst = a_addr + ((q & 1) ? dst_odd : dst_even) + q * (kRowsPerInstr * kRowBytes);
            const char* src = src_kb + static_cast<long long>(row > 0 ? row : 0) * pitch_bytes;
            cp_async16(dst, src, row >= 0 ? 16u : 0u);
          }
        }
        // the stage's "rows landed" barrier fires by itself when this thread's copies are done, so a
        // stage becomes usable as soon as its data is there, whatever this thread waits for next
        cp_async_arrive_noinc(smem_u32(&ctl->afull[s]));
      }
    };
    // Four index registers, each reloaded right after its stage has been issued and not
    // touched again until four stages later: the loads stay in flight across the stages between.
    int nid0, nid1, nid2, nid3, kp0, kp1, kp2, kp3;
    load_stage(g0, nid0, kp0);
    load_stage(g0 + 1, nid1, kp1);
    load_stage(g0 + 2, nid2, kp2);
    load_stage(g0 + 3, nid3, kp3);
    if (ls.settled) asm volatile("griddepcontrol.wait;" ::: "memory");
    for (int g = g0; g < g1 && ok; g += 4) {
      run_stage(nid0, kp0);
      load_stage(g + 4, nid0, kp0);
      if (g + 1 < g1 && ok) run_stage(nid1, kp1);
      load_stage(g + 5, nid1, kp1);
      if (g + 2 < g1 && ok) run_stage(nid2, kp2);
      load_stage(g + 6, nid2, kp2);
      if (g + 3 < g1 && ok) run_stage(nid3, kp3);
      load_stage(g + 7, nid3, kp3);
    }
    } else {
    // ---- several offsets per stage (cin = 64 / SLOTS channels each) ----
    constexpr int kSlotChunks = 8 / SLOTS;  // 16-byte chunks of one slot inside the 128-byte row
    const int my_slot = chunk / kSlotChunks, my_cc = chunk % kSlotChunks;
    auto load_stage = [&](int g, int (&nid)[SLOTS], int (&kp)[SLOTS]) {
#pragma unroll
      for (int q = 0; q < SLOTS; ++q) {
        nid[q] = -1;
        kp[q] = -2;
        if (g < g1) {
          nid[q] = __ldg(ls.stage_nbr + (static_cast<size_t>(g) * SLOTS + q) * kRows + tid);
          kp[q] = __ldg(ls.stage_kp + static_cast<size_t>(g) * SLOTS + q);
        }
      }
    };
    auto run_stage = [&](const int (&nid)[SLOTS], const int (&kp)[SLOTS]) {
      const bool second = kp[0] == -1;  // the identity stage: slot 0 only, the second operand's width
      const int nkb = second ? kblocks2 : 1;
      for (int kb = 0; kb < nkb; ++kb, ++j) {
        const int s = j % kStages;
        const int n = j / kStages;
        if (n > 0) ok = mbar_wait(smem_u32(&ctl->empty[s]), (n - 1) & 1, ctl);
        ok = __all_sync(0xFFFFFFFFu, ok);
        if (!ok) return;
        const uint32_t a_addr = tiles_addr + s * stage_bytes;
        const uint32_t b_addr = a_addr + kAStage;
        if (second) {
          if (warp == 0 && elect_one()) {
            const uint32_t bbar = smem_u32(&ctl->bfull[s]);
            mbar_arrive_expect_tx(bbar, b_bytes);
            bulk_copy_g2s(b_addr, sec.w2 + static_cast<size_t>(kb) * cout * 64, b_bytes, bbar);
          }
          const int kchunks = min(8, (sec.cin2 - kb * 64) >> 3);
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            const int r = q * 4 + rsub;
            const int src_row = __shfl_sync(0xFFFFFFFFu, nid[0], r);
            if (chunk < kchunks) {
              const uint32_t dst = a_addr + (warp * 32 + r) * 128 + ((chunk ^ (r & 7)) << 4);
              const __half* src = sec.in2 + (src_row >= 0 ? static_cast<size_t>(src_row) * sec.cin2 + kb * 64 + chunk * 8 : 0);
              cp_async16(dst, src, src_row >= 0 ? 16u : 0u);
            }
          }
        } else {
          if (tid == 0) mbar_arrive(smem_u32(&ctl->bfull[s]));  // the weights below ride on afull; keep bfull's phase in step
          // weight block: per slot the offset's [cout][cin] image, chunk by chunk into the swizzled
          // K-major block; unused slots are zero-filled so that the MMA can always run all K steps
          // (chunk ch of output channel co's 128-byte row belongs to slot ch / kSlotChunks: no run-time division)
          for (int c = tid; c < cout * 8; c += kRows) {
            const int co = c >> 3, ch = c & 7;
            const int q = ch / kSlotChunks, cc = ch % kSlotChunks;
            int kq = kp[0];
#pragma unroll
            for (int u = 1; u < SLOTS; ++u) kq = q == u ? kp[u] : kq;
            const uint32_t dst = b_addr + co * 128 + ((ch ^ (co & 7)) << 4);
            const __half* src = ls.wslots + (kq >= 0 ? (static_cast<size_t>(kq) * cout + co) * cin + cc * 8 : 0);
            cp_async16(dst, src, kq >= 0 ? 16u : 0u);
          }
          const char* src_lane = reinterpret_cast<const char*>(in) + my_cc * 16;
          const int pitch_bytes = ep.ld_in * 2;
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            const int r = q * 4 + rsub;
            int src_row = -1;
#pragma unroll
            for (int u = 0; u < SLOTS; ++u) {
              const int v = __shfl_sync(0xFFFFFFFFu, nid[u], r);
              if (u == my_slot) src_row = v;
            }
            const uint32_t dst = a_addr + ((q & 1) ? dst_odd : dst_even) + q * (4 * 128);
            const char* src = src_lane + static_cast<long long>(src_row > 0 ? src_row : 0) * pitch_bytes;
            cp_async16(dst, src, src_row >= 0 ? 16u : 0u);
          }
        }
        cp_async_arrive_noinc(smem_u32(&ctl->afull[s]));
      }
    };
    // two stages of indices in flight (SLOTS entries each)
    int nidA[SLOTS], kpA[SLOTS], nidB[SLOTS], kpB[SLOTS];
    load_stage(g0, nidA, kpA);
    load_stage(g0 + 1, nidB, kpB);
    if (ls.settled) asm volatile("griddepcontrol.wait;" ::: "memory");
    for (int g = g0; g < g1 && ok; g += 2) {
      run_stage(nidA, kpA);
      load_stage(g + 2, nidA, kpA);
      if (g + 1 < g1 && ok) run_stage(nidB, kpB);
      load_stage(g + 3, nidB, kpB);
    }
    }
    cp_async_wait_all();
    if (!ok && tid == 0) {
      // aborting: give this thread's bulk copies a bounded chance to land before the CTA leaves
      for (int u = max(0, j - kStages); u < j; ++u) {
        const uint32_t bar = smem_u32(&ctl->bfull[u % kStages]);
        for (int spin = 0; spin < (1 << 20) && !mbar_try_wait(bar, (u / kStages) & 1); ++spin) {
        }
      }
    }
  } else if (warp == kMmaWarp) {
    // =========================== MMA issuer ===========================
    if (ls.settled) asm volatile("griddepcontrol.wait;" ::: "memory");
    {
      const uint32_t idesc = (1u << 4) | (static_cast<uint32_t>(cout >> 3) << 17) | (static_cast<uint32_t>(kTileM >> 4) << 24);
      int j = 0;
      bool ok = true;
      first_bounds();
      for (int t = t0; t < t1 && ok; ++t) {
        const int it = t - t0;
        const int buf = it % nacc;
        const Work work = next_work(t);
        const int nst_main = work.main;
        const int nst = nst_main + (work.ident ? kblocks2 : 0);
        // the accumulator must have been drained by the epilogue (two tiles ago)
        if (it >= nacc) ok = mbar_wait(smem_u32(&ctl->accempty[buf]), ((it / nacc) - 1) & 1, ctl);
        ok = __all_sync(0xFFFFFFFFu, ok);
        if (!ok) break;
        tc_fence_after();
        const uint32_t tmem_acc = tmem_base + static_cast<uint32_t>(buf * SUB * cout);
        uint32_t accumulate = 0;
        int kb = 0;  // K block inside the offset
        for (int st = 0; st < nst; ++st, ++j) {
          const int s = j % kStages;
          const uint32_t par = (j / kStages) & 1;
          ok = mbar_wait(smem_u32(&ctl->afull[s]), par, ctl) && mbar_wait(smem_u32(&ctl->bfull[s]), par, ctl);
          ok = __all_sync(0xFFFFFFFFu, ok);
          if (!ok) break;
          const bool second = st >= nst_main;
          if (st == nst_main) kb = 0;
          if (elect_one()) {
            fence_proxy_async();  // the gathered rows were written through the generic proxy
            tc_fence_after();
            const uint32_t a_addr = tiles_addr + s * stage_bytes;
            const uint64_t db = make_desc(a_addr + kAStage);
            // with several offsets per stage the whole 64-channel block is always filled (unused slots with zeros)
            const int ksteps = (SLOTS > 1 && !second) ? 4 : min(KB / 16, ((second ? sec.cin2 : cin) - kb * KB) >> 4);
#pragma unroll
            for (int k = 0; k < KB / 16; ++k) {
              if (k < ksteps) {
#pragma unroll
                for (int sub = 0; sub < SUB; ++sub) {  // the same weight block feeds every sub-tile
                  const uint64_t da = make_desc(a_addr + sub * (kTileM * kRowBytes));
                  tc_mma_f16(tmem_acc + static_cast<uint32_t>(sub * cout), da + static_cast<uint64_t>(k * 2),
                             db + static_cast<uint64_t>(k * 2), idesc, k > 0 ? 1u : accumulate);
                }
              }
            }
            tc_commit(smem_u32(&ctl->empty[s]));
          }
          __syncwarp();
          accumulate = 1;
          if (++kb == kblocks && !second) kb = 0;
        }
        if (!ok) break;
        if (elect_one()) {
          if (nst > 0)
            tc_commit(smem_u32(&ctl->accfull[buf]));  // arrives when every MMA of the tile has finished
          else
            mbar_arrive(smem_u32(&ctl->accfull[buf]));  // no MMA was issued: the epilogue writes zeros
        }
        __syncwarp();
      }
    }
    __syncwarp();
    tc_fence_before();
  } else {
    // =========================== epilogue ===========================
    const int lane_quarter = warp & 3;  // the TMEM lanes this warp may read: 32*(warp%4)..+31
    const int slot_in_tile = lane_quarter * 32 + lane;
    // every 16-channel piece of an output row is 32-byte aligned: one 256-bit store per piece
    const bool wide_out = (ep.ld_out & 15) == 0 && (reinterpret_cast<uintptr_t>(out) & 31) == 0;
    const bool wide_res = (reinterpret_cast<uintptr_t>(ep.residual) & 31) == 0;  // (rows of C_out = 16k channels)
    if (ls.settled) asm volatile("griddepcontrol.wait;" ::: "memory");
    first_bounds();
    for (int t = t0; t < t1; ++t) {
      const int it = t - t0;
      const Work work = next_work(t);
      const int buf = it % nacc;
      int rows_of[SUB];
#pragma unroll
      for (int sub = 0; sub < SUB; ++sub) {
        const int slot = t * kRows + sub * kTileM + slot_in_tile;
        rows_of[sub] = n_out;
        if (slot < n_out) rows_of[sub] = ls.order ? __ldg(ls.order + slot) : slot;
      }
      const bool any = work.main + (work.ident ? kblocks2 : 0) > 0;
      const bool cut = work.cut;
      if (ep.residual) {
        // the rows are known before the accumulator is: pull the residual rows into L2 while waiting
#pragma unroll
        for (int sub = 0; sub < SUB; ++sub) {
          if (rows_of[sub] < n_out) {
            const char* rp = reinterpret_cast<const char*>(ep.residual + static_cast<size_t>(rows_of[sub]) * cout);
            for (int off = 0; off < cout * 2; off += 64) asm volatile("prefetch.global.L2 [%0];" ::"l"(rp + off));
          }
        }
      }
      bool ok = mbar_wait(smem_u32(&ctl->accfull[buf]), (it / nacc) & 1, ctl);
      ok = __all_sync(0xFFFFFFFFu, ok);
      if (!ok) break;
      tc_fence_after();
      // last tile of this CTA: once every CTA is here (or gone), the next kernel of the stream may be
      // set up on the SMs; it waits for this grid's completion before it touches memory
      if (t == t1 - 1) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
      if (parts > 1) {  // (one tile per CTA; its sums stay in tensor memory until the cluster adds them up below)
        part_any = any;
        break;
      }
#pragma unroll
      for (int sub = 0; sub < SUB; ++sub) {
      const int my_row = rows_of[sub];
      const bool store_row = my_row < n_out;
      const uint32_t taddr = tmem_base + static_cast<uint32_t>((buf * SUB + sub) * cout) +
                             (static_cast<uint32_t>(lane_quarter * 32) << 16);
      __half* orow = out + static_cast<size_t>(store_row ? my_row : 0) * ep.ld_out;
      __half* prow[2] = {nullptr, nullptr};
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        if (PUSH && ep.push_slot[s] && store_row) {
          const int slot = __ldg(ep.push_slot[s] + my_row);
          if (slot >= 0) prow[s] = ep.push_base[s] + static_cast<size_t>(slot) * cout;
        }
      }
      const __half* rrow = (ep.residual && store_row) ? ep.residual + static_cast<size_t>(my_row) * cout : nullptr;
      for (int c0 = 0; c0 < cout; c0 += 16) {
        uint4 ra = make_uint4(0u, 0u, 0u, 0u), rb = ra;
        if (rrow) {  // issued ahead of the tensor-memory load, consumed after it
          if (wide_res) {
            load32(rrow + c0, ra, rb);
          } else {
            ra = *reinterpret_cast<const uint4*>(rrow + c0);
            rb = *reinterpret_cast<const uint4*>(rrow + c0 + 8);
          }
        }
        uint32_t r[16];
        if (any) {  // warp-uniform: the tensor-memory load is warp-collective
          tmem_ld16(taddr + c0, r);
          tmem_ld_wait();
        } else {
#pragma unroll
          for (int q = 0; q < 16; ++q) r[q] = 0u;
        }
        float v[16];
#pragma unroll
        for (int q = 0; q < 16; ++q) v[q] = __uint_as_float(r[q]);
        if (cut) {  // a piece of a tile cut between CTAs: k_sum_cut_tiles adds the pieces
          float4* dst = reinterpret_cast<float4*>(
              ep.partial + ((static_cast<size_t>(blockIdx.x) * 2 + (t == t0 ? 0 : 1)) * kTileM + slot_in_tile) * cout + c0);
#pragma unroll
          for (int q = 0; q < 4; ++q) dst[q] = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
          continue;
        }
        if (ep.scale || ep.shift) {
#pragma unroll
          for (int q = 0; q < 16; q += 4) {
            const float4 s4 = *reinterpret_cast<const float4*>(affine + c0 + q);
            const float4 t4 = *reinterpret_cast<const float4*>(affine + cout + c0 + q);
            v[q] = fmaf(v[q], s4.x, t4.x);
            v[q + 1] = fmaf(v[q + 1], s4.y, t4.y);
            v[q + 2] = fmaf(v[q + 2], s4.z, t4.z);
            v[q + 3] = fmaf(v[q + 3], s4.w, t4.w);
          }
        }
        if (rrow) {
          const __half2* ha = reinterpret_cast<const __half2*>(&ra);
          const __half2* hb = reinterpret_cast<const __half2*>(&rb);
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const float2 fa = __half22float2(ha[q]);
            const float2 fb = __half22float2(hb[q]);
            v[2 * q] += fa.x;
            v[2 * q + 1] += fa.y;
            v[8 + 2 * q] += fb.x;
            v[8 + 2 * q + 1] += fb.y;
          }
        }
        uint4 oa, ob;
        __half2* pa = reinterpret_cast<__half2*>(&oa);
        __half2* pb = reinterpret_cast<__half2*>(&ob);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          pa[q] = __floats2half2_rn(act_apply(v[2 * q], ep.act, ep.slope), act_apply(v[2 * q + 1], ep.act, ep.slope));
          pb[q] = __floats2half2_rn(act_apply(v[8 + 2 * q], ep.act, ep.slope),
                                    act_apply(v[8 + 2 * q + 1], ep.act, ep.slope));
        }
        if (store_row) {
          if (wide_out) {
            store32(orow + c0, oa, ob);
          } else {
            *reinterpret_cast<uint4*>(orow + c0) = oa;
            *reinterpret_cast<uint4*>(orow + c0 + 8) = ob;
          }
        }
#pragma unroll
        for (int s = 0; s < 2; ++s) {
          if (PUSH && prow[s]) {
            *reinterpret_cast<uint4*>(prow[s] + c0) = oa;
            *reinterpret_cast<uint4*>(prow[s] + c0 + 8) = ob;
          }
        }
      }
      }  // sub-tiles
      tc_fence_before();
      mbar_arrive(smem_u32(&ctl->accempty[buf]));  // 128 arrivals hand the accumulator back
    }
    tc_fence_before();
  }
  if constexpr (SUB == 1 && SLOTS == 1 && !PUSH) {
    if (parts > 1) {
      // The parts' sums, added up through the cluster's shared memory.  The ring is idle by now (the accumulator is
      // complete, so every stage has been consumed): as many columns as fit it at a time, column groups of four
      // outermost, so that lanes (rows) touch consecutive 16 bytes.  Part p finishes rows p * 128 / parts on.  Against
      // sums through global memory and a second kernel: 256->256 on 7.5 k rows, four parts, 40 -> 28 us.
      const int part = static_cast<int>(blockIdx.x) % parts;
      const int fit = (kStages * stage_bytes / (kTileM * 4)) & ~15;
      const int rows_each = kTileM / parts;
      const bool scaled = ep.scale || ep.shift;
      for (int base = 0; base < cout; base += fit) {
        const int cols = min(fit, cout - base);
        __syncthreads();
        if (warp > kMmaWarp) {
          const int r = (warp & 3) * 32 + lane;
          const uint32_t taddr = tmem_base + static_cast<uint32_t>(base) + (static_cast<uint32_t>((warp & 3) * 32) << 16);
          for (int c0 = 0; c0 < cols; c0 += 16) {
            uint32_t v[16];
            if (part_any) {
              tmem_ld16(taddr + c0, v);
              tmem_ld_wait();
            } else {
#pragma unroll
              for (int q = 0; q < 16; ++q) v[q] = 0u;
            }
            uint4* dst = reinterpret_cast<uint4*>(tiles) + (c0 / 4) * kTileM + r;
#pragma unroll
            for (int q = 0; q < 4; ++q) dst[q * kTileM] = make_uint4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
          }
        }
        tc_fence_before();
        cluster_sync();
        for (int i = tid; i < rows_each * (cols / 8); i += 32 * (4 * SUB + 5)) {
          const int r = part * rows_each + i % rows_each, c0 = i / rows_each * 8;
          const int slot = t0 * kTileM + r;
          if (slot >= n_out) continue;
          const int row = ls.order ? __ldg(ls.order + slot) : slot;
          const uint32_t src = tiles_addr + static_cast<uint32_t>((c0 / 4) * kTileM + r) * 16u;
          float v[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
          for (int p = 0; p < parts; ++p) {
            const float4 x = cluster_ld4(src, p), y = cluster_ld4(src + kTileM * 16u, p);
            v[0] += x.x; v[1] += x.y; v[2] += x.z; v[3] += x.w;
            v[4] += y.x; v[5] += y.y; v[6] += y.z; v[7] += y.w;
          }
          const int c = base + c0;
          if (scaled) {
#pragma unroll
            for (int q = 0; q < 8; ++q) v[q] = fmaf(v[q], affine[c + q], affine[cout + c + q]);
          }
          finish8(v, row, c, cout, out, ep);
        }
        cluster_sync();  // (the other parts have read this CTA's sums)
      }
    }
  }
  __syncthreads();
  if (warp == kMmaWarp) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base),
                 "r"(static_cast<uint32_t>(tmem_cols))
                 : "memory");
  }
}


// =====================================================================================================
// k_conv_umma_mt: several accumulators per CTA, offsets taken in offset-major order, row ring and weight
// ring decoupled.
//
// A super-tile is SUB (1, 2 or 4) consecutive 128-row sub-tiles of the processing order, each with its own
// accumulator in tensor memory.  The tile lists of a super-tile name every offset that any of its rows has,
// with a presence bit per sub-tile (stage_kp bits 8..).  Per listed offset and 64-channel K block the weight
// block is staged ONCE (weight ring, nb slots of C_out x 128 B, one bulk async copy each) and multiplied
// with the gathered rows of every sub-tile that has the offset (row ring, na slots of 128 rows x 128 B).
// Against one ring stage = rows + weights per (128-row tile, offset) this
//   * divides the weight traffic from L2 by the number of sub-tiles that share an offset (rows are sorted
//     by indicator bitmask, so neighbouring sub-tiles share most of theirs), and
//   * frees the shared memory that every stage spent on its own weight copy for row slots: what limits
//     the fused kernel is the number of row gathers in flight per SM (a ring slot is occupied for about
//     3 us from the first copy instruction to the release by the tensor core).
// Warps: 4*SUB producers (one thread per row of the super-tile; the four warps of a sub-tile fill that
// sub-tile's row slots), one MMA warp (one lane issues), one weight-loader warp (one lane), 4*EPIW
// epilogue warps (EPIW teams; team e drains the accumulators of sub-tiles e, e+EPIW, ..).  All follow the
// same sequence: stage g of the super-tile, K block kb, present sub-tiles in ascending order.  Every
// sub-tile has its OWN ring of na row slots: a slot is then filled and released by the same warps in
// strict alternation, which the parity waits of mbarriers need (a ring shared between sub-tiles lets a
// sub-tile that skipped a use of a slot run two phases ahead of its barrier, where the parity test
// passes wrongly).  With nsets = 2 the accumulators alternate between super-tiles, so the epilogue
// of super-tile i overlaps the products of i+1.  Same bounded waits, abort protocol, programmatic dependent
// launch and epilogue as k_conv_umma; results are bit-identical to it (same products, same order per row).
constexpr int kMaxA = 16;
constexpr int kMaxB = 4;
constexpr int kMaxAcc = 8;

struct SharedCtlMt {
  unsigned long long afull[kMaxA];
  unsigned long long aempty[kMaxA];
  unsigned long long bfull[kMaxB];
  unsigned long long bempty[kMaxB];
  unsigned long long accfull[kMaxAcc];
  unsigned long long accempty[kMaxAcc];
  uint32_t tmem_base;
  int range[2];
  volatile int abort_flag;
};

// stage_kp entry -> (offset or -1 for the identity stage, presence mask over the sub-tiles)
template <int SUB>
__device__ __forceinline__ void decode_stage(int code, int& kp, uint32_t& present) {
  constexpr uint32_t kAll = (1u << SUB) - 1u;
  if (code < 0) {
    kp = code;
    present = code == -1 ? kAll : 0u;
    return;
  }
  kp = code & 255;
  present = (static_cast<uint32_t>(code) >> 8) & kAll;
  if (present == 0u) present = kAll;  // lists without presence bits: every sub-tile takes part
}

template <int SUB, int EPIW>
__global__ void __launch_bounds__(32 * (4 * SUB + 2 + 4 * EPIW), SUB == 1 ? 2 : 1)
    k_conv_umma_mt(const __half* __restrict__ in, const __half* __restrict__ wpacked, Lists ls, Second sec, int n_out, int cin,
                   int cout, __half* __restrict__ out, Epi ep, int tmem_cols, int na, int nb, int nsets) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_addr = smem_u32(smem_raw);
  const uint32_t pad = ((raw_addr + 1023u) & ~1023u) - raw_addr;
  uint8_t* tiles = smem_raw + pad;  // 1024-byte aligned
  const uint32_t a_base = raw_addr + pad;
  const int b_bytes = cout * 128;
  const uint32_t b_base = a_base + static_cast<uint32_t>(SUB * na) * kABytes;  // na row slots per sub-tile
  constexpr int kRows = kTileM * SUB;
  constexpr int kProd = 4 * SUB;  // producer warps
  constexpr int kMmaWarp = kProd;
  constexpr int kLoadWarp = kProd + 1;
  SharedCtlMt* ctl =
      reinterpret_cast<SharedCtlMt*>(tiles + static_cast<size_t>(SUB * na) * kABytes + static_cast<size_t>(nb) * b_bytes);

  const int tid = threadIdx.x;
  const int warp = tid >> 5;
  const int lane = tid & 31;
  const int kblocks = (cin + 63) >> 6;
  const int kblocks2 = sec.in2 ? (sec.cin2 + 63) >> 6 : 0;
  const int n_tiles = (n_out + kRows - 1) / kRows;

  if (tid == 0) {
    for (int s = 0; s < SUB * na; ++s) {
      mbar_init(smem_u32(&ctl->afull[s]), kTileM);
      mbar_init(smem_u32(&ctl->aempty[s]), 1);
    }
    for (int s = 0; s < nb; ++s) {
      mbar_init(smem_u32(&ctl->bfull[s]), 1);
      mbar_init(smem_u32(&ctl->bempty[s]), 1);
    }
    for (int s = 0; s < kMaxAcc; ++s) {
      mbar_init(smem_u32(&ctl->accfull[s]), 1);
      mbar_init(smem_u32(&ctl->accempty[s]), 128);
    }
    ctl->abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == kMmaWarp) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&ctl->tmem_base)),
                 "r"(static_cast<uint32_t>(tmem_cols))
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (!ls.settled) asm volatile("griddepcontrol.wait;" ::: "memory");
  if (warp < 2) {
    const int unit = kblocks > 1 ? 2 : 1;
    const long long total = cost_before(ls.tile_ptr, n_tiles, unit);
    const unsigned b = blockIdx.x + warp;
    const int t = b >= gridDim.x ? n_tiles : warp_tile_at_cost(ls.tile_ptr, n_tiles, total * b / gridDim.x, unit, lane);
    if (lane == 0) ctl->range[warp] = t;
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = ctl->tmem_base;
  const int t0 = ctl->range[0], t1 = ctl->range[1];
  const int g0 = __ldg(ls.tile_ptr + t0), g1 = __ldg(ls.tile_ptr + t1);

  if (warp < kProd) {
    // =========================== row producers ===========================
    const int sub = warp >> 2;          // this warp's sub-tile
    const int row_in_sub = tid & 127;   // this thread's row inside it
    const int wq = warp & 3;            // warp inside the sub-tile
    const int rsub = lane >> 3;         // row inside a 4-row group
    const int chunk = lane & 7;         // 16-byte chunk inside a 128-byte row
    const int ring0 = sub * na;  // this sub-tile's own row slots: ring0 .. ring0 + na - 1
    int js = 0;                  // row items this sub-tile has produced so far
    bool ok = true;
    auto load_stage = [&](int g, int& nid, int& code) {
      nid = -1;
      code = -2;
      if (g < g1) {
        code = __ldg(ls.stage_kp + g);
        int kp;
        uint32_t present;
        decode_stage<SUB>(code, kp, present);
        if ((present >> sub) & 1u) nid = __ldg(ls.stage_nbr + static_cast<size_t>(g) * kRows + sub * kTileM + row_in_sub);
      }
    };
    auto run_stage = [&](int nid, int code) {
      int kp;
      uint32_t present;
      decode_stage<SUB>(code, kp, present);
      if (!((present >> sub) & 1u)) return;
      const bool second = kp == -1;
      const int nkb = second ? kblocks2 : kblocks;
      const __half* src_base = second ? sec.in2 : in;
      const int width = second ? sec.cin2 : cin;
      const int pitch = second ? sec.cin2 : ep.ld_in;
      for (int kb = 0; kb < nkb; ++kb, ++js) {
        const int s = ring0 + js % na;
        const int n = js / na;
        if (n > 0) ok = mbar_wait(smem_u32(&ctl->aempty[s]), (n - 1) & 1, ctl, 1 | (sub << 4), js);
        ok = __all_sync(0xFFFFFFFFu, ok);  // keep the warp convergent for the shuffles below
        if (!ok) return;
        const uint32_t a_addr = a_base + static_cast<uint32_t>(s) * kABytes;
        const int kchunks = min(8, (width - kb * 64) >> 3);
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          const int r = q * 4 + rsub;  // row inside this warp's 32
          const int src_row = __shfl_sync(0xFFFFFFFFu, nid, r);
          if (chunk < kchunks) {
            const uint32_t dst = a_addr + (wq * 32 + r) * 128 + ((chunk ^ (r & 7)) << 4);
            const __half* src = src_base + (src_row >= 0 ? static_cast<size_t>(src_row) * pitch + kb * 64 + chunk * 8 : 0);
            cp_async16(dst, src, src_row >= 0 ? 16u : 0u);
          }
        }
        cp_async_arrive_noinc(smem_u32(&ctl->afull[s]));
      }
    };
    int nid0, nid1, nid2, nid3, c0, c1, c2, c3;
    load_stage(g0, nid0, c0);
    load_stage(g0 + 1, nid1, c1);
    load_stage(g0 + 2, nid2, c2);
    load_stage(g0 + 3, nid3, c3);
    if (ls.settled) asm volatile("griddepcontrol.wait;" ::: "memory");
    for (int g = g0; g < g1 && ok; g += 4) {
      run_stage(nid0, c0);
      load_stage(g + 4, nid0, c0);
      if (g + 1 < g1 && ok) run_stage(nid1, c1);
      load_stage(g + 5, nid1, c1);
      if (g + 2 < g1 && ok) run_stage(nid2, c2);
      load_stage(g + 6, nid2, c2);
      if (g + 3 < g1 && ok) run_stage(nid3, c3);
      load_stage(g + 7, nid3, c3);
    }
    cp_async_wait_all();
  } else if (warp == kLoadWarp) {
    // =========================== weight loader ===========================
    if (ls.settled) asm volatile("griddepcontrol.wait;" ::: "memory");
    if (lane == 0) {
      int jb = 0;
      bool ok = true;
      for (int g = g0; g < g1 && ok; ++g) {
        int kp;
        uint32_t present;
        decode_stage<SUB>(__ldg(ls.stage_kp + g), kp, present);
        const bool second = kp == -1;
        const int nkb = second ? kblocks2 : kblocks;
        if (present == 0u) continue;
        for (int kb = 0; kb < nkb; ++kb, ++jb) {
          const int s = jb % nb;
          const int n = jb / nb;
          if (n > 0) ok = mbar_wait(smem_u32(&ctl->bempty[s]), (n - 1) & 1, ctl, 2, jb);
          if (!ok) break;
          const uint32_t bbar = smem_u32(&ctl->bfull[s]);
          mbar_arrive_expect_tx(bbar, b_bytes);
          const __half* wsrc = second ? sec.w2 + static_cast<size_t>(kb) * cout * 64
                                      : wpacked + (static_cast<size_t>(kp) * kblocks + kb) * cout * 64;
          bulk_copy_g2s(b_base + static_cast<uint32_t>(s) * b_bytes, wsrc, b_bytes, bbar);
        }
      }
      if (!ok) {
        // aborting: give the bulk copies in flight a bounded chance to land before the CTA leaves
        for (int u = max(0, jb - nb); u < jb; ++u) {
          const uint32_t bar = smem_u32(&ctl->bfull[u % nb]);
          for (int spin = 0; spin < (1 << 20) && !mbar_try_wait(bar, (u / nb) & 1); ++spin) {
          }
        }
      }
    }
    __syncwarp();
  } else if (warp == kMmaWarp) {
    // =========================== MMA issuer ===========================
    if (ls.settled) asm volatile("griddepcontrol.wait;" ::: "memory");
    if (lane == 0) {
      const uint32_t idesc = (1u << 4) | (static_cast<uint32_t>(cout >> 3) << 17) | (static_cast<uint32_t>(kTileM >> 4) << 24);
      int jb = 0;
      int js[SUB];  // row items consumed so far, per sub-tile
#pragma unroll
      for (int sub = 0; sub < SUB; ++sub) js[sub] = 0;
      bool ok = true;
      for (int t = t0; t < t1 && ok; ++t) {
        const int it = t - t0;
        const int set = it % nsets;
        const uint32_t acc_par = static_cast<uint32_t>((it / nsets) - 1) & 1u;  // phase of the previous use's release
        uint32_t touched = 0u;
        const int ga = __ldg(ls.tile_ptr + t), gb = __ldg(ls.tile_ptr + t + 1);
        for (int g = ga; g < gb && ok; ++g) {
          int kp;
          uint32_t present;
          decode_stage<SUB>(__ldg(ls.stage_kp + g), kp, present);
          const bool second = kp == -1;
          const int nkb = second ? kblocks2 : kblocks;
          if (present == 0u) continue;
          for (int kb = 0; kb < nkb && ok; ++kb, ++jb) {
            const int bs = jb % nb;
            ok = mbar_wait(smem_u32(&ctl->bfull[bs]), (jb / nb) & 1, ctl, 3 | (it << 8), jb);
            if (!ok) break;
            const uint64_t db = make_desc(b_base + static_cast<uint32_t>(bs) * b_bytes);
            const int ksteps = min(4, ((second ? sec.cin2 : cin) - kb * 64) >> 4);
#pragma unroll
            for (int sub = 0; sub < SUB; ++sub) {
              if (!((present >> sub) & 1u)) continue;
              const int acc = set * SUB + sub;
              if (!((touched >> sub) & 1u) && it >= nsets) {
                // first product into this accumulator: its previous contents must have been drained
                ok = mbar_wait(smem_u32(&ctl->accempty[acc]), acc_par, ctl, 4 | (sub << 4) | (it << 8), js[sub]);
                if (!ok) break;
              }
              const int as = sub * na + js[sub] % na;
              ok = mbar_wait(smem_u32(&ctl->afull[as]), (js[sub] / na) & 1, ctl, 5 | (sub << 4) | (it << 8), js[sub]);
              if (!ok) break;
              fence_proxy_async();  // the gathered rows were written through the generic proxy
              tc_fence_after();
              const uint64_t da = make_desc(a_base + static_cast<uint32_t>(as) * kABytes);
              const uint32_t tmem_acc = tmem_base + static_cast<uint32_t>(acc * cout);
              for (int k = 0; k < ksteps; ++k)
                tc_mma_f16(tmem_acc, da + static_cast<uint64_t>(k * 2), db + static_cast<uint64_t>(k * 2), idesc,
                           (((touched >> sub) & 1u) || k > 0) ? 1u : 0u);
              touched |= 1u << sub;
              tc_commit(smem_u32(&ctl->aempty[as]));
              ++js[sub];
            }
            if (!ok) break;
            tc_commit(smem_u32(&ctl->bempty[bs]));
          }
        }
        if (!ok) break;
#pragma unroll
        for (int sub = 0; sub < SUB; ++sub) {
          const int acc = set * SUB + sub;
          if ((touched >> sub) & 1u) {
            tc_commit(smem_u32(&ctl->accfull[acc]));  // arrives when every product issued so far has finished
          } else {
            // nothing went into this accumulator: the epilogue writes zeros.  The signal may still not
            // run two phases ahead of the epilogue, so the previous use's release is waited for here too.
            if (it >= nsets) ok = mbar_wait(smem_u32(&ctl->accempty[acc]), acc_par, ctl, 6 | (sub << 4) | (it << 8), jb);
            if (!ok) break;
            mbar_arrive(smem_u32(&ctl->accfull[acc]));
          }
        }
      }
    }
    __syncwarp();
    tc_fence_before();
  } else {
    // =========================== epilogue ===========================
    const int e = warp - (kProd + 2);
    const int team = e >> 2;
    const int lane_quarter = warp & 3;  // the TMEM lanes this warp may read: 32*(warp%4)..+31
    const int slot_in_sub = lane_quarter * 32 + lane;
    if (ls.settled) asm volatile("griddepcontrol.wait;" ::: "memory");
    bool ok = true;
    for (int t = t0; t < t1 && ok; ++t) {
      const int it = t - t0;
      const int set = it % nsets;
      // which accumulators of this super-tile received products: OR of the stages' presence masks
      uint32_t any_mask = 0u;
      {
        const int ga = __ldg(ls.tile_ptr + t), gb = __ldg(ls.tile_ptr + t + 1);
        for (int g = ga + lane; g < gb; g += 32) {
          int kp;
          uint32_t present;
          decode_stage<SUB>(__ldg(ls.stage_kp + g), kp, present);
          if (kp == -1 && kblocks2 == 0) present = 0u;  // identity stage listed, but no second operand in this launch
          any_mask |= present;
        }
        any_mask = __reduce_or_sync(0xFFFFFFFFu, any_mask);
      }
      if (t == t1 - 1) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
      for (int sub = team; sub < SUB && ok; sub += EPIW) {
        const int acc = set * SUB + sub;
        const int slot = t * kRows + sub * kTileM + slot_in_sub;
        int my_row = n_out;
        if (slot < n_out) my_row = ls.order ? __ldg(ls.order + slot) : slot;
        const bool store_row = my_row < n_out;
        const bool any = (any_mask >> sub) & 1u;
        if (ep.residual && store_row) {
          const char* rp = reinterpret_cast<const char*>(ep.residual + static_cast<size_t>(my_row) * cout);
          for (int off = 0; off < cout * 2; off += 64) asm volatile("prefetch.global.L2 [%0];" ::"l"(rp + off));
        }
        ok = mbar_wait(smem_u32(&ctl->accfull[acc]), (it / nsets) & 1, ctl, 7 | (sub << 4) | (it << 8), t);
        ok = __all_sync(0xFFFFFFFFu, ok);
        if (!ok) break;
        tc_fence_after();
        const uint32_t taddr = tmem_base + static_cast<uint32_t>(acc * cout) + (static_cast<uint32_t>(lane_quarter * 32) << 16);
        __half* orow = out + static_cast<size_t>(store_row ? my_row : 0) * ep.ld_out;
        const __half* rrow = (ep.residual && store_row) ? ep.residual + static_cast<size_t>(my_row) * cout : nullptr;
        for (int c0 = 0; c0 < cout; c0 += 16) {
          uint4 ra = make_uint4(0u, 0u, 0u, 0u), rb = ra;
          if (rrow) {  // issued ahead of the tensor-memory load, consumed after it
            ra = *reinterpret_cast<const uint4*>(rrow + c0);
            rb = *reinterpret_cast<const uint4*>(rrow + c0 + 8);
          }
          uint32_t r[16];
          if (any) {  // warp-uniform: the tensor-memory load is warp-collective
            tmem_ld16(taddr + c0, r);
            tmem_ld_wait();
          } else {
#pragma unroll
            for (int q = 0; q < 16; ++q) r[q] = 0u;
          }
          float v[16];
#pragma unroll
          for (int q = 0; q < 16; ++q) v[q] = __uint_as_float(r[q]);
          if (ep.scale || ep.shift) {  // one fused multiply-add per value, as in k_conv_umma (bit-identical results)
#pragma unroll
            for (int q = 0; q < 16; q += 4) {
              const float4 s4 = ep.scale ? __ldg(reinterpret_cast<const float4*>(ep.scale + c0 + q)) : make_float4(1.f, 1.f, 1.f, 1.f);
              const float4 t4 = ep.shift ? __ldg(reinterpret_cast<const float4*>(ep.shift + c0 + q)) : make_float4(0.f, 0.f, 0.f, 0.f);
              v[q] = fmaf(v[q], s4.x, t4.x);
              v[q + 1] = fmaf(v[q + 1], s4.y, t4.y);
              v[q + 2] = fmaf(v[q + 2], s4.z, t4.z);
              v[q + 3] = fmaf(v[q + 3], s4.w, t4.w);
            }
          }
          if (rrow) {
            const __half2* ha = reinterpret_cast<const __half2*>(&ra);
            const __half2* hb = reinterpret_cast<const __half2*>(&rb);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              const float2 fa = __half22float2(ha[q]);
              const float2 fb = __half22float2(hb[q]);
              v[2 * q] += fa.x;
              v[2 * q + 1] += fa.y;
              v[8 + 2 * q] += fb.x;
              v[8 + 2 * q + 1] += fb.y;
            }
          }
          uint4 oa, ob;
          __half2* pa = reinterpret_cast<__half2*>(&oa);
          __half2* pb = reinterpret_cast<__half2*>(&ob);
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            pa[q] = __floats2half2_rn(act_apply(v[2 * q], ep.act, ep.slope), act_apply(v[2 * q + 1], ep.act, ep.slope));
            pb[q] = __floats2half2_rn(act_apply(v[8 + 2 * q], ep.act, ep.slope),
                                      act_apply(v[8 + 2 * q + 1], ep.act, ep.slope));
          }
          if (store_row) {
            *reinterpret_cast<uint4*>(orow + c0) = oa;
            *reinterpret_cast<uint4*>(orow + c0 + 8) = ob;
          }
        }
        tc_fence_before();
        mbar_arrive(smem_u32(&ctl->accempty[acc]));  // 128 arrivals hand the accumulator back
      }
    }
    tc_fence_before();
  }
  __syncthreads();
  if (warp == kMmaWarp) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base),
                 "r"(static_cast<uint32_t>(tmem_cols))
                 : "memory");
  }
}

// =====================================================================================================
// k_conv_deep: the same layer with ONE CTA per SM, its rows gathered by the TMA engine.
//
// What bounds k_conv_umma on layers of one offset per stage is instruction latency: a producer warp needs 1000 to 1400 cycles
// for a stage (index shuffles, eight row copies, barrier), the MMA warp 400 to 700 for its four products, and a copy
// that only fills in zeros takes three times as long as one that moves data.  Here
//   * rows come by tile::gather4, four rows per operation.  One operation costs the issuing warp 80 cycles, which made
//     it look slow from one warp (2576 cycles for a stage's 128 rows); sixteen warps that issue half a stage each keep
//     the L2 port busy (240 cycles a stage, 68 of about 71 bytes per clock and SM) and do nothing else.  The data arrives
//     through the async proxy: nobody has to order it before the products.
//   * groups of four rows that all lack the offset are not copied: the warp stores zeros, once for as long as the same
//     group of the slot stays without rows (an out-of-range row costs the TMA engine 40 cycles);
//   * one thread issues the products in a short loop over running descriptors.  Unrolled over the ring, with every slot's
//     descriptors and barriers known up to their base, a stage is cheaper by itself (230 to 300 cycles against 400 to 700),
//     but that code, like an epilogue that carries every option through every tile, does not fit the instruction caches
//     beside the other roles': layers took up to twice as long;
//   * the SM's shared memory is one ring of 4 to 9 stages, and two teams of epilogue warps take the tiles in turn with two
//     or four accumulators between them: no product waits for a tile's stores;
//   * a third as many CTAs have shares three times as long, against which the heaviest tiles (27 offsets, where the mean is
//     2 to 5) weigh less.
// Kernel only, us, k_conv_umma / this: 64->64 on 200 k rows of a room 29.9 / 22.3, 96->96 on 240 k rows of four scans 45.9 / 38.3,
// 256->256 on 1.5 M rows 544 / 502, 64->64 5x5x5 on 1.5 M rows 408 / 278.  What bounds it now: with 256 channels the round trip of a
// ring of four 48 KB stages (41 bytes per clock and SM from L2, tensor pipe half busy); with few, the heaviest CTA's chain of
// stages and the set-up of a layer (about 4 us to the first product).
// Lists, shares of tiles, second operand, split tiles and bounded waits are k_conv_umma's.  Widths are multiples of
// 32 input channels (the last 32 of an odd multiple are a half block, as there).
constexpr int kDeepMaxRing = 9;
constexpr int kDeepMaxAcc = 4;
constexpr int kDeepTeams = 2;
constexpr int kDeepWide = 128;  // output channels from which a tile's columns are shared by the teams
constexpr int kDeepMmaWarp = 4 * kDeepTeams;   // epilogue warps first: warp & 3 is a warp's quarter of tensor memory
constexpr int kDeepProducers = kDeepMmaWarp + 1;
constexpr int kDeepBounds = 184;               // tile bounds of a CTA kept in shared memory (more cost 96 and 128 channels a stage)
// producer warps per slot: each fills its part of the slot's rows
constexpr int deep_parts(int ring) { return ring == 4 ? 4 : 2; }
constexpr int deep_threads(int ring) { return 32 * (kDeepProducers + ring * deep_parts(ring)); }

struct DeepMaps {
  CUtensorMap in;     // [n_in][cin], boxes of one row x 64 channels
  CUtensorMap in32;   // boxes of 32 channels (the half block)
  CUtensorMap sec;    // the second operand's
  CUtensorMap sec32;
};

struct DeepCtl {
  unsigned long long full[kDeepMaxRing];
  unsigned long long empty[kDeepMaxRing];
  unsigned long long accfull[kDeepMaxAcc];
  unsigned long long accempty[kDeepMaxAcc];
  uint32_t tmem_base;
  int range[2];
  volatile int abort_flag;
  int bounds[kDeepBounds];
};

// Rows r.x .. r.w (negative: zeros) of the map's box at column x, one after the other from dst on.
__device__ __forceinline__ void gather4(uint32_t dst, const CUtensorMap* map, int x, const int4& r, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cta.global.tile::gather4.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5, %6}], [%7];" ::"r"(dst),
      "l"(map), "r"(x), "r"(r.x), "r"(r.y), "r"(r.z), "r"(r.w), "r"(bar)
      : "memory");
}

template <bool HALF, int RING>
__global__ void __launch_bounds__(deep_threads(RING), 1)
    k_conv_deep(const __grid_constant__ DeepMaps maps, const __half* __restrict__ wpacked, const Lists ls, const Second sec, int n_out,
                int cin, int cout, __half* __restrict__ out, const Epi ep, int tmem_cols, int nacc) {
  constexpr int PARTS = deep_parts(RING), kPartRows = kTileM / PARTS, kQuads = kPartRows / 4;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_addr = smem_u32(smem_raw);
  const uint32_t pad = ((raw_addr + 1023u) & ~1023u) - raw_addr;
  uint8_t* tiles = smem_raw + pad;  // 1024-byte aligned
  const uint32_t tiles_addr = raw_addr + pad;
  constexpr int KB = 64;
  const int b_bytes = cout * 128;
  const int stage_bytes = kABytes + b_bytes;
  DeepCtl* ctl = reinterpret_cast<DeepCtl*>(tiles + RING * stage_bytes);
  float* affine = reinterpret_cast<float*>(ctl + 1);
  static_assert(sizeof(DeepCtl) % 16 == 0, "the staged scale/shift are read as float4");
  const bool wide = cout >= kDeepWide;  // both teams take half of every tile's columns
  const int tid = threadIdx.x;
  const int warp = tid >> 5;
  const int lane = tid & 31;
  const int kblocks = (cin + KB - 1) / KB;
  const int kblocks2 = sec.in2 ? (sec.cin2 + KB - 1) / KB : 0;
  const int tall = ls.tall, n_tiles = (n_out + (kTileM << tall) - 1) >> (7 + tall);  // the lists' tiles
  if (tid == 0) {
    for (int s = 0; s < RING; ++s) {
      mbar_init(smem_u32(&ctl->full[s]), PARTS);
      mbar_init(smem_u32(&ctl->empty[s]), 1);
    }
    for (int s = 0; s < nacc; ++s) {
      mbar_init(smem_u32(&ctl->accfull[s]), 1);
      mbar_init(smem_u32(&ctl->accempty[s]), wide ? 256 : 128);
    }
    ctl->abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp < kDeepMmaWarp && (ep.scale || ep.shift)) {
    for (int c = tid; c < cout; c += 32 * kDeepMmaWarp) {
      affine[c] = ep.scale ? __ldg(ep.scale + c) : 1.f;
      affine[cout + c] = ep.shift ? __ldg(ep.shift + c) : 0.f;
    }
  }
  if (warp == kDeepMmaWarp) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&ctl->tmem_base)),
                 "r"(static_cast<uint32_t>(tmem_cols))
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (!ls.settled) asm volatile("griddepcontrol.wait;" ::: "memory");  // (as in k_conv_umma)
  const int parts = ep.parts > 1 ? ep.parts : 1;
  if (parts > 1) {
    if (tid == 0) {
      ctl->range[0] = static_cast<int>(blockIdx.x) / parts;
      ctl->range[1] = static_cast<int>(blockIdx.x) / parts + 1;
    }
  } else if (static_cast<int>(gridDim.x) == n_tiles) {  // a tile each
    if (tid < 2) ctl->range[tid] = static_cast<int>(blockIdx.x) + tid;
  } else if (warp < 2) {
    // a tile's stores cost about two ring stages: 64->64 on 200 k rows 20.7 us so, 22.9 with one, 28.3 with a quarter; 5x5x5 on
    // 300 k rows 110, 129, 140; 96->96 on 240 k rows 36 so, 44 with four
    const int unit = kblocks, fixed = 2;
    const long long total = cost_before(ls.tile_ptr, n_tiles, unit, fixed);
    const unsigned b = blockIdx.x + warp;
    const int t = b >= gridDim.x ? n_tiles : warp_tile_at_cost(ls.tile_ptr, n_tiles, total * b / gridDim.x, unit, lane, fixed);
    if (lane == 0) ctl->range[warp] = t;
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = ctl->tmem_base;
  const int first_tile = ctl->range[0], last_tile = ctl->range[1];
  for (int i = tid; i <= last_tile - first_tile && i < kDeepBounds; i += deep_threads(RING))
    ctl->bounds[i] = first_stage(ls.tile_ptr, first_tile + i);
  __syncthreads();
  const int t0 = first_tile << tall, t1 = min(last_tile << tall, (n_out + kTileM - 1) / kTileM);  // in tiles of 128 rows
  auto bound = [&](int t) { return t - first_tile < kDeepBounds ? ctl->bounds[t - first_tile] : first_stage(ls.tile_ptr, t); };
  struct Work {
    int first;        // first entry of the lists (of this CTA's part)
    int main, ident;  // ring stages of the listed offsets; with the identity stage
  };
  auto work_of = [&](int t) {
    const int b0 = bound(t >> tall), b1 = bound((t >> tall) + 1);
    int sa = b0, sb = b1;
    if (parts > 1) {
      const int n = sb - sa, part = static_cast<int>(blockIdx.x) % parts;
      const int a = sa + static_cast<int>(static_cast<long long>(n) * part / parts);
      sb = sa + static_cast<int>(static_cast<long long>(n) * (part + 1) / parts);
      sa = a;
    }
    Work w;
    w.first = sa * ls.entries;
    w.ident = (ls.identity && sb > sa && sb == b1) ? 1 : 0;
    w.main = (sb - sa - w.ident) * ls.entries * kblocks;
    return w;
  };

  bool part_any = false;
  if (warp >= kDeepProducers) {
    // =========================== producers: warp p fills part p % PARTS of slot p / PARTS, use after use ===========================
    const int slot = (warp - kDeepProducers) / PARTS, part = (warp - kDeepProducers) % PARTS;
    const uint32_t a_part = tiles_addr + slot * stage_bytes + part * kPartRows * 128;  // (half blocks: rows of 64 bytes)
    const uint32_t full = smem_u32(&ctl->full[slot]), empty = smem_u32(&ctl->empty[slot]);
    const unsigned inv = ((1u << 20) + kblocks - 1) / kblocks;  // stage / kblocks of a tile's at most 128 x kblocks stages
    int t = t0, before = 0, j = slot;  // `before`: ring stages in front of tile t; j: the slot's next stage
    Work w = {0, 0, 0};
    int in_tile = 0;
    if (t < t1) {
      w = work_of(t);
      in_tile = w.main + (w.ident ? kblocks2 : 0);
    }
    int4 rows = make_int4(-1, -1, -1, -1);
    int kb = 0, kp = 0;
    bool second = false;
    auto fetch = [&]() -> bool {  // the slot's next stage: its rows (asked for) and what they are multiplied with
      while (t < t1 && j >= before + in_tile) {
        before += in_tile;
        if (++t < t1) {
          w = work_of(t);
          in_tile = w.main + (w.ident ? kblocks2 : 0);
        }
      }
      if (t >= t1) return false;
      const int i = j - before;
      second = i >= w.main;
      const int o = static_cast<int>((static_cast<unsigned>(second ? w.main : i) * inv) >> 20);
      kb = second ? i - w.main : i - o * kblocks;
      const int g = w.first + o;
      if (lane < kQuads) {
        if (ls.tile_ptr) {
          rows = __ldg(reinterpret_cast<const int4*>(ls.stage_nbr + (static_cast<size_t>(g) << (7 + tall)) + ((t & tall) * kTileM + part * kPartRows)) + lane);
        } else {
          const int r = g * kTileM + part * kPartRows + 4 * lane;
          rows = make_int4(r < n_out ? r : -1, r + 1 < n_out ? r + 1 : -1, r + 2 < n_out ? r + 2 : -1, r + 3 < n_out ? r + 3 : -1);
        }
      }
      if (part == 0 && ls.tile_ptr && !second) {
        kp = __ldg(ls.stage_kp + g);
        kp = kp < 0 ? 0 : kp & 255;  // (negative: an entry without an offset, no rows; bits 8..: sub-tile presence)
      }
      j += RING;
      return true;
    };
    bool ok = true, was_half = false;
    uint32_t use = 0, zeroed = 0;  // zeroed: groups of the part that hold zeros
    bool more = fetch();
    if (ls.settled) asm volatile("griddepcontrol.wait;" ::: "memory");
    while (more) {
      // (the copies below read rows, kb, kp and second; the next stage is fetched behind them)
      const int nkb = second ? kblocks2 : kblocks;
      const bool half = HALF && kb == nkb - 1 && (second ? sec.wtail : ls.wtail) != nullptr;
      const int quad_bytes = half ? 256 : 512;
      const uint32_t a_addr = half ? tiles_addr + slot * stage_bytes + part * kPartRows * 64 : a_part;
      const bool any = lane < kQuads && (rows.x & rows.y & rows.z & rows.w) >= 0;  // (a row that is there has no sign bit)
      const uint32_t gathered = __ballot_sync(0xFFFFFFFFu, any);
      if (use > 0) ok = mbar_wait(empty, (use - 1) & 1, ctl);
      ok = __all_sync(0xFFFFFFFFu, ok);
      if (!ok) break;
      constexpr uint32_t kAll = kQuads == 32 ? 0xFFFFFFFFu : (1u << kQuads) - 1u;
      const uint32_t blank = kAll & ~gathered;
      if (half != was_half) zeroed = 0;  // (another layout)
      was_half = half;
      const uint32_t fill = blank & ~zeroed;
      if (fill) {
        for (uint32_t m = fill; m; m &= m - 1u) {
          const uint32_t at = a_addr + (__ffs(m) - 1) * quad_bytes + lane * 16;
          if (lane * 16 < quad_bytes) asm volatile("st.shared.v4.b32 [%0], {%1, %1, %1, %1};" ::"r"(at), "r"(0) : "memory");
        }
        fence_proxy_async();  // plain stores, read by the tensor core
        __syncwarp();
      }
      zeroed = blank;
      if (elect_one()) {
        const uint32_t row_bytes = static_cast<uint32_t>(__popc(gathered) * quad_bytes);
        if (part == 0) {
          const uint32_t w_bytes = half ? static_cast<uint32_t>(cout) * 64u : static_cast<uint32_t>(b_bytes);
          mbar_arrive_expect_tx(full, row_bytes + w_bytes);
          const __half* wtail = second ? sec.wtail : ls.wtail;
          const __half* wsrc = second ? sec.w2 + static_cast<size_t>(kb) * cout * KB
                                      : wpacked + (static_cast<size_t>(kb) + static_cast<size_t>(kp) * kblocks) * cout * KB;
          if (half) wsrc = wtail + (static_cast<size_t>(second ? 0 : kp) * (2 * nkb - 1) + 2 * kb) * cout * 32;
          bulk_copy_g2s(tiles_addr + slot * stage_bytes + kABytes, wsrc, w_bytes, full);
        } else {
          mbar_arrive_expect_tx(full, row_bytes);
        }
      }
      __syncwarp();
      if (any) gather4(a_addr + lane * quad_bytes, second ? (half ? &maps.sec32 : &maps.sec) : (half ? &maps.in32 : &maps.in), kb * KB, rows, full);
      ++use;
      more = fetch();
    }
    if (!ok && use > 0 && lane == 0) {
      // aborting: give the slot's copies a bounded chance to land before the CTA leaves
      for (int spin = 0; spin < (1 << 20) && !mbar_try_wait(full, (use - 1) & 1); ++spin) {
      }
    }
  } else if (warp == kDeepMmaWarp) {
    // =========================== MMA issuer: one thread ===========================
    if (ls.settled) asm volatile("griddepcontrol.wait;" ::: "memory");
    if (elect_one()) {
      const uint32_t idesc = (1u << 4) | (static_cast<uint32_t>(cout >> 3) << 17) | (static_cast<uint32_t>(kTileM >> 4) << 24);
      const uint32_t lo0 = (tiles_addr >> 4) | (1u << 16), step = static_cast<uint32_t>(stage_bytes) >> 4;
      constexpr uint32_t kHi = (1024u >> 4) | (1u << 14) | (2u << 29), kHi32 = (512u >> 4) | (1u << 14) | (4u << 29);
      // (kHi: make_desc; kHi32: half blocks, rows of 64 B, 64-byte swizzle, 8-row groups 512 B apart)
      const int last1 = ((cin - 1) & 63) / 16 + 1, last2 = ((sec.cin2 - 1) & 63) / 16 + 1;  // K steps of the last K block
      const uint32_t full0 = smem_u32(&ctl->full[0]), empty0 = smem_u32(&ctl->empty[0]);
      uint32_t par = 0, lo = lo0, at = 0;  // at: 8 x the slot
      bool ok = true;
      for (int t = t0; t < t1 && ok; ++t) {
        const Work work = work_of(t);
        const int round = (t - t0) >> (nacc == 4 ? 2 : 1), buf = (t - t0) & (nacc - 1);
        const uint32_t acc = tmem_base + static_cast<uint32_t>(buf * cout);
        if (round > 0) ok = mbar_wait(smem_u32(&ctl->accempty[buf]), (round - 1) & 1, ctl);
        uint32_t accumulate = 0;
        auto blocks = [&](int n, int nkb, int last, bool half_end) {  // n stages, nkb to an offset
          int kb = nkb;
          for (; n > 0 && ok; --n) {
            ok = mbar_wait(full0 + at, par, ctl);
            if (!ok) break;
            tc_fence_after();
            if (--kb > 0 || (last == 4 && !half_end)) {
              tc_mma_f16_lohi(acc, lo, kHi, lo + (kABytes >> 4), kHi, idesc, accumulate);
              tc_mma_f16_lohi(acc, lo + 2, kHi, lo + (kABytes >> 4) + 2, kHi, idesc, 1u);
              tc_mma_f16_lohi(acc, lo + 4, kHi, lo + (kABytes >> 4) + 4, kHi, idesc, 1u);
              tc_mma_f16_lohi(acc, lo + 6, kHi, lo + (kABytes >> 4) + 6, kHi, idesc, 1u);
            } else if (half_end) {
              tc_mma_f16_lohi(acc, lo, kHi32, lo + (kABytes >> 4), kHi32, idesc, accumulate);
              tc_mma_f16_lohi(acc, lo + 2, kHi32, lo + (kABytes >> 4) + 2, kHi32, idesc, 1u);
            } else {
              for (int k = 0; k < last; ++k)
                tc_mma_f16_lohi(acc, lo + 2 * k, kHi, lo + (kABytes >> 4) + 2 * k, kHi, idesc, k > 0 ? 1u : accumulate);
            }
            tc_commit(empty0 + at);
            accumulate = 1;
            if (kb == 0) kb = nkb;
            at += 8;
            lo += step;
            if (at == 8 * RING) {
              at = 0;
              lo = lo0;
              par ^= 1;
            }
          }
        };
        if (!ok) break;
        tc_fence_after();
        blocks(work.main, kblocks, last1, HALF && ls.wtail);
        if (work.ident && kblocks2) blocks(kblocks2, kblocks2, last2, HALF && sec.wtail);
        if (!ok) break;
        if (work.main > 0 || (work.ident && kblocks2))
          tc_commit(smem_u32(&ctl->accfull[buf]));  // arrives when every MMA of the tile has finished
        else
          mbar_arrive(smem_u32(&ctl->accfull[buf]));  // no MMA was issued: the epilogue writes zeros
      }
    }
    __syncwarp();
    tc_fence_before();
  } else {
    // =========================== epilogue ===========================
    const int team = warp >> 2;
    const int lane_quarter = warp & 3;
    const int slot_in_tile = lane_quarter * 32 + lane;
    const bool wide_out = (ep.ld_out & 15) == 0 && (reinterpret_cast<uintptr_t>(out) & 31) == 0;
    const bool wide_res = (reinterpret_cast<uintptr_t>(ep.residual) & 31) == 0;
    const bool scaled = ep.scale || ep.shift;
    const bool plain = wide_out && !scaled && !ep.residual && ep.act == PCE_ACT_NONE;
    const bool folded = wide_out && scaled && !ep.residual && ep.act == PCE_ACT_RELU;
    auto row_of = [&](int t) {
      const int slot = t * kTileM + slot_in_tile;
      return t < t1 && slot < n_out ? (ls.order ? __ldg(ls.order + slot) : slot) : n_out;
    };
    // Two teams: a tile each in turn, or (wide outputs, and a CTA with one tile) half the columns each of every tile, which ends
    // the last tile sooner: 256 columns of a tile take one team about 8000 cycles.
    const bool halves = wide || t1 - t0 == 1;
    const int c_mid = halves ? (cout / 2 + 15) & ~15 : 0, c_from = team ? c_mid : 0, c_to = halves && !team ? c_mid : cout;
    const int t_step = halves ? 1 : kDeepTeams, t_first = halves ? t0 : t0 + team;
    int my_row = row_of(t_first);
    if (ls.settled) asm volatile("griddepcontrol.wait;" ::: "memory");
    for (int t = t_first; t < t1; t += t_step) {
      const int it = t - t0;
      const Work work = work_of(t);
      const int buf = it & (nacc - 1), round = it / nacc;
      const bool store_row = my_row < n_out;
      const bool any = work.main + (work.ident ? kblocks2 : 0) > 0;
      __half* orow = out + static_cast<size_t>(store_row ? my_row : 0) * ep.ld_out;
      const __half* rrow = (ep.residual && store_row) ? ep.residual + static_cast<size_t>(my_row) * cout : nullptr;
      my_row = row_of(t + t_step);  // (a tile ahead)
      if (rrow) {
        // the rows are known before the accumulator is: pull the residual rows into L2 while waiting
        const char* rp = reinterpret_cast<const char*>(rrow);
        for (int off = 0; off < cout * 2; off += 64) asm volatile("prefetch.global.L2 [%0];" ::"l"(rp + off));
      }
      bool ok = mbar_wait(smem_u32(&ctl->accfull[buf]), round & 1, ctl);
      ok = __all_sync(0xFFFFFFFFu, ok);
      if (!ok) break;
      tc_fence_after();
      if (t == t1 - 1) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
      if (parts > 1) {  // (one tile per CTA; its sums stay in tensor memory until the cluster adds them up below)
        part_any = any;
        break;
      }
      const uint32_t taddr = tmem_base + static_cast<uint32_t>(buf * cout) + (static_cast<uint32_t>(lane_quarter * 32) << 16);
      if (plain && any) {
        // nothing but the conversion: kept apart, since the code of all the other cases, stepped over or predicated off, took
        // longer to fetch than this takes to run
        int c0 = c_from;
#pragma unroll 1
        for (; c0 + 32 <= c_to; c0 += 32) {
          uint32_t r[32];
          tmem_ld32(taddr + c0, r);
          tmem_ld_wait();
          uint4 o[4];
          uint32_t* po = reinterpret_cast<uint32_t*>(o);
#pragma unroll
          for (int q = 0; q < 16; ++q) po[q] = pack_half2(r[2 * q], r[2 * q + 1]);
          if (store_row) {
            store32(orow + c0, o[0], o[1]);
            store32(orow + c0 + 16, o[2], o[3]);
          }
        }
        if (c0 < c_to) {
          uint32_t r[16];
          tmem_ld16(taddr + c0, r);
          tmem_ld_wait();
          uint4 o[2];
          uint32_t* po = reinterpret_cast<uint32_t*>(o);
#pragma unroll
          for (int q = 0; q < 8; ++q) po[q] = pack_half2(r[2 * q], r[2 * q + 1]);
          if (store_row) store32(orow + c0, o[0], o[1]);
        }
      } else if (folded && any) {
        // a folded BatchNorm and ReLU: what most layers of a network have
#pragma unroll 1
        for (int c0 = c_from; c0 < c_to; c0 += 16) {
          uint32_t r[16];
          tmem_ld16(taddr + c0, r);
          tmem_ld_wait();
          uint4 o[2];
          uint32_t* po = reinterpret_cast<uint32_t*>(o);
#pragma unroll
          for (int q = 0; q < 16; q += 4) {
            const float4 s4 = *reinterpret_cast<const float4*>(affine + c0 + q);
            const float4 t4 = *reinterpret_cast<const float4*>(affine + cout + c0 + q);
            // (a NaN becomes zero, as in the general form)
            const float a = fmaxf(fmaf(__uint_as_float(r[q]), s4.x, t4.x), 0.f), b = fmaxf(fmaf(__uint_as_float(r[q + 1]), s4.y, t4.y), 0.f);
            const float c = fmaxf(fmaf(__uint_as_float(r[q + 2]), s4.z, t4.z), 0.f), d = fmaxf(fmaf(__uint_as_float(r[q + 3]), s4.w, t4.w), 0.f);
            po[q / 2] = pack_half2(__float_as_uint(a), __float_as_uint(b));
            po[q / 2 + 1] = pack_half2(__float_as_uint(c), __float_as_uint(d));
          }
          if (store_row) store32(orow + c0, o[0], o[1]);
        }
      } else
#pragma unroll 1
      for (int c0 = c_from; c0 < c_to; c0 += 16) {
        uint4 ra, rb;
        if (rrow) {  // issued ahead of the tensor-memory load, consumed after it
          if (wide_res) {
            load32(rrow + c0, ra, rb);
          } else {
            ra = *reinterpret_cast<const uint4*>(rrow + c0);
            rb = *reinterpret_cast<const uint4*>(rrow + c0 + 8);
          }
        }
        uint32_t r[16];
        if (any) {  // warp-uniform: the tensor-memory load is warp-collective
          tmem_ld16(taddr + c0, r);
          tmem_ld_wait();
        } else {
#pragma unroll
          for (int q = 0; q < 16; ++q) r[q] = 0u;
        }
        float v[16];
#pragma unroll
        for (int q = 0; q < 16; ++q) v[q] = __uint_as_float(r[q]);
        if (scaled) {
#pragma unroll
          for (int q = 0; q < 16; q += 4) {
            const float4 s4 = *reinterpret_cast<const float4*>(affine + c0 + q);
            const float4 t4 = *reinterpret_cast<const float4*>(affine + cout + c0 + q);
            v[q] = fmaf(v[q], s4.x, t4.x);
            v[q + 1] = fmaf(v[q + 1], s4.y, t4.y);
            v[q + 2] = fmaf(v[q + 2], s4.z, t4.z);
            v[q + 3] = fmaf(v[q + 3], s4.w, t4.w);
          }
        }
        if (rrow) {
          const __half2* ha = reinterpret_cast<const __half2*>(&ra);
          const __half2* hb = reinterpret_cast<const __half2*>(&rb);
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const float2 fa = __half22float2(ha[q]);
            const float2 fb = __half22float2(hb[q]);
            v[2 * q] += fa.x;
            v[2 * q + 1] += fa.y;
            v[8 + 2 * q] += fb.x;
            v[8 + 2 * q + 1] += fb.y;
          }
        }
        if (ep.act == PCE_ACT_RELU) {
#pragma unroll
          for (int q = 0; q < 16; ++q) v[q] = v[q] > 0.f ? v[q] : 0.f;
        } else if (ep.act == PCE_ACT_LEAKY) {
#pragma unroll
          for (int q = 0; q < 16; ++q) v[q] = v[q] > 0.f ? v[q] : v[q] * ep.slope;
        }
        uint4 oa, ob;
        __half2* pa = reinterpret_cast<__half2*>(&oa);
        __half2* pb = reinterpret_cast<__half2*>(&ob);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          pa[q] = __floats2half2_rn(v[2 * q], v[2 * q + 1]);
          pb[q] = __floats2half2_rn(v[8 + 2 * q], v[8 + 2 * q + 1]);
        }
        if (store_row) {
          if (wide_out) {
            store32(orow + c0, oa, ob);
          } else {
            *reinterpret_cast<uint4*>(orow + c0) = oa;
            *reinterpret_cast<uint4*>(orow + c0 + 8) = ob;
          }
        }
      }
      tc_fence_before();
      mbar_arrive(smem_u32(&ctl->accempty[buf]));  // 128 arrivals hand the accumulator back
    }
    tc_fence_before();
  }
  if (parts > 1) {
    // the parts' sums, added up through the cluster's shared memory as in k_conv_umma
    const int part = static_cast<int>(blockIdx.x) % parts;
    // (the ring holds them all: four stages' weight blocks alone are 512 bytes a column)
    static_assert(RING >= 4, "room for 128 rows of fp32 sums");
    const int rows_each = kTileM / parts;
    const bool scaled = ep.scale || ep.shift;
    __syncthreads();
    if (warp < 4) {
      const int r = warp * 32 + lane;
      const uint32_t taddr = tmem_base + (static_cast<uint32_t>(warp * 32) << 16);
      for (int c0 = 0; c0 < cout; c0 += 16) {
        uint32_t v[16];
        if (part_any) {
          tmem_ld16(taddr + c0, v);
          tmem_ld_wait();
        } else {
#pragma unroll
          for (int q = 0; q < 16; ++q) v[q] = 0u;
        }
        uint4* dst = reinterpret_cast<uint4*>(tiles) + (c0 / 4) * kTileM + r;
#pragma unroll
        for (int q = 0; q < 4; ++q) dst[q * kTileM] = make_uint4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
      }
    }
    tc_fence_before();
    cluster_sync();
    for (int i = tid; i < rows_each * (cout / 8); i += deep_threads(RING)) {
      const int r = part * rows_each + i % rows_each, c0 = i / rows_each * 8;
      const int slot = t0 * kTileM + r;
      if (slot >= n_out) continue;
      const int row = ls.order ? __ldg(ls.order + slot) : slot;
      const uint32_t src = tiles_addr + static_cast<uint32_t>((c0 / 4) * kTileM + r) * 16u;
      float v[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      for (int p = 0; p < parts; ++p) {
        const float4 x = cluster_ld4(src, p), y = cluster_ld4(src + kTileM * 16u, p);
        v[0] += x.x; v[1] += x.y; v[2] += x.z; v[3] += x.w;
        v[4] += y.x; v[5] += y.y; v[6] += y.z; v[7] += y.w;
      }
      if (scaled) {
#pragma unroll
        for (int q = 0; q < 8; ++q) v[q] = fmaf(v[q], affine[c0 + q], affine[cout + c0 + q]);
      }
      finish8(v, row, c0, cout, out, ep);
    }
    cluster_sync();  // (the other parts have read this CTA's sums)
  }
  __syncthreads();
  if (warp == kDeepMmaWarp) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base),
                 "r"(static_cast<uint32_t>(tmem_cols))
                 : "memory");
  }
}

// Second kernel of a stream-K layer: for every tile that was cut between CTAs, adds the pieces in CTA order
// (fp32) and applies the epilogue; tiles that one CTA finished are left alone.  Block (x, t) handles 256 of the
// tile's (row, 8 output channels) items: its first warp works out which CTAs hold pieces of tile t (consecutive
// CTAs, one per lane, 32 per round; the divisions are done once per block, not per item), then every thread sums
// its item over them.  `ctas` = the grid of the convolution launch.
__global__ void __launch_bounds__(256)
    k_sum_cut_tiles(const float* __restrict__ partial, const int* __restrict__ tile_ptr, const int* __restrict__ order,
                    int n_tiles, int ctas, int n_out, int cout, __half* __restrict__ out, Epi ep) {
  __shared__ int s_slot[32];  // per CTA of the round: 2*b + which, or -1 (its share misses the tile)
  __shared__ int s_whole;     // some CTA held the whole tile: nothing to do
  asm volatile("griddepcontrol.wait;" ::: "memory");  // launched while the convolution kernel drains
  const int t = blockIdx.y;
  const int a = __ldg(tile_ptr + t), e = __ldg(tile_ptr + t + 1);
  const long long total = __ldg(tile_ptr + n_tiles);
  const int chunks = cout >> 3;
  const int item = static_cast<int>(blockIdx.x) * 256 + static_cast<int>(threadIdx.x);
  const bool live = item < kTileM * chunks;
  const int r = live ? item / chunks : 0, c0 = live ? (item % chunks) * 8 : 0;
  // CTAs that can hold stages of [a, e): b with share_begin(b) < e and share_begin(b + 1) > a
  int b0 = 0, b1 = -1;
  if (e > a && total > 0) {
    b0 = static_cast<int>(static_cast<long long>(a) * ctas / total) - 1;
    b1 = static_cast<int>(static_cast<long long>(e) * ctas / total) + 1;
    b0 = b0 < 0 ? 0 : b0;
    b1 = b1 > ctas - 1 ? ctas - 1 : b1;
  }
  if (threadIdx.x == 0) s_whole = 0;
  float v[8];
#pragma unroll
  for (int q = 0; q < 8; ++q) v[q] = 0.f;
  for (int base = b0; base <= b1; base += 32) {
    __syncthreads();
    if (threadIdx.x < 32) {
      const int b = base + static_cast<int>(threadIdx.x);
      int slot = -1;
      if (b <= b1) {
        const int sb = share_begin(total, b, ctas), se = share_begin(total, b + 1, ctas);
        if ((sb > a ? sb : a) < (se < e ? se : e)) {
          if (sb <= a && se >= e) s_whole = 1;
          slot = 2 * b + (sb >= a ? 0 : 1);  // the tile is the CTA's first tile when its share starts inside it
        }
      }
      s_slot[threadIdx.x] = slot;
    }
    __syncthreads();
    if (s_whole) return;
    if (live) {
      for (int k = 0; k < 32; ++k) {
        const int slot = s_slot[k];
        if (slot < 0) continue;
        const float4* src = reinterpret_cast<const float4*>(partial + (static_cast<size_t>(slot) * kTileM + r) * cout + c0);
        const float4 x = __ldg(src), y = __ldg(src + 1);
        v[0] += x.x; v[1] += x.y; v[2] += x.z; v[3] += x.w;
        v[4] += y.x; v[5] += y.y; v[6] += y.z; v[7] += y.w;
      }
    }
  }
  // (a tile without stages belongs to no share: its rows get the epilogue of zero here)
  const int slot_row = t * kTileM + r;
  if (!live || slot_row >= n_out) return;
  const int row = order ? __ldg(order + slot_row) : slot_row;
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    if (ep.scale || ep.shift)
      v[q] = fmaf(v[q], ep.scale ? __ldg(ep.scale + c0 + q) : 1.f, ep.shift ? __ldg(ep.shift + c0 + q) : 0.f);
  }
  finish8(v, row, c0, cout, out, ep);
}

}  // namespace umma

bool conv_umma_supported(int cin, int cout, int dtype) {
  return dtype == PCE_F16 && cin >= 16 && cin % 16 == 0 && cout >= 16 && cout % 16 == 0 && cout <= 256;
}

// Per-offset blocks, and for 16 or 32 input channels also the per-offset [cout][cin] images from which
// stages that hold several offsets assemble their weight block.
// Behind them, a second copy as 32-channel blocks (cout rows x 64 B, 64-byte swizzle) for widths that are an odd
// multiple of 32 (their last K block is half, see HALF) and for every single-offset weight (a second
// operand of such a layer).
static bool has_kb32_image(int kv, int cin) { return kv == 1 || cin % 64 == 32; }
static size_t kb64_image_bytes(int kv, int cin, int cout) {
  const size_t blocks = static_cast<size_t>(kv) * ((cin + 63) / 64) * cout * 128;
  return blocks + ((cin == 16 || cin == 32) ? static_cast<size_t>(kv) * cout * cin * 2 : 0);
}
size_t umma_packed_bytes(int kv, int cin, int cout) {
  const size_t kb32 = has_kb32_image(kv, cin) ? static_cast<size_t>(kv) * ((cin + 31) / 32) * cout * 64 : 0;
  return kb64_image_bytes(kv, cin, cout) + kb32;
}

int umma_pack_weights(const void* w, int kv, int cin, int cout, void* packed, cudaStream_t st) {
  const int kblocks = (cin + 63) / 64;
  const long long total = static_cast<long long>(kv) * kblocks * cout * 64;
  const int grid = static_cast<int>(std::min<long long>((total + 255) / 256, 148ll * 8));
  umma::k_pack_weights<<<grid, 256, 0, st>>>(static_cast<const __half*>(w), kv, cin, cout, kblocks,
                                             static_cast<__half*>(packed), 64);
  PCE_LAUNCH_CHECK();
  if (has_kb32_image(kv, cin)) {
    const int kblocks32 = (cin + 31) / 32;
    const long long total32 = static_cast<long long>(kv) * kblocks32 * cout * 32;
    umma::k_pack_weights<<<static_cast<int>(std::min<long long>((total32 + 255) / 256, 148ll * 8)), 256, 0, st>>>(
        static_cast<const __half*>(w), kv, cin, cout, kblocks32,
        reinterpret_cast<__half*>(static_cast<char*>(packed) + kb64_image_bytes(kv, cin, cout)), 32);
    PCE_LAUNCH_CHECK();
  }
  if (cin == 16 || cin == 32) {
    const long long n = static_cast<long long>(kv) * cout * cin;
    umma::k_pack_weight_slots<<<static_cast<int>(std::min<long long>((n + 255) / 256, 148ll * 8)), 256, 0, st>>>(
        static_cast<const __half*>(w), kv, cin, cout, static_cast<__half*>(packed) + total);
    PCE_LAUNCH_CHECK();
  }
  return PCE_OK;
}

// Tuning hooks (tests / experiments): 0 = choose; stages 2..4; sub-tiles 1 or 2; accumulator sets 1 or 2.
int umma_force_stages = 0;
int umma_force_sub = 0;
int umma_force_nacc = 0;
// Programmatic dependent launch: the kernel's set-up (barriers, tensor-memory allocation; with settled
// tile lists also the tile search and the first index loads) overlaps the tail of the kernel before it
// in the stream.  0 = off, 1 = on, 2 = on but every list is treated as not settled.
int umma_overlap_launches = 1;
// 1: layers with one offset per stage and no halo push run k_conv_umma_mt (several accumulators per CTA,
// decoupled row and weight rings); 0 (default): k_conv_umma, which measured faster at every tile height
// both kernels share (512-row tiles exist for k_conv_umma_mt only and always run on it).
int umma_multi_tile = 0;

template <int SUB, int EPIW>
static void launch_umma_mt(int grid, size_t smem, cudaStream_t st, const __half* in, const __half* w, const umma::Lists& ls,
                           const umma::Second& sec, int n_out, int cin, int cout, __half* out, const umma::Epi& e,
                           int tmem_cols, int na, int nb, int nsets) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(32 * (4 * SUB + 2 + 4 * EPIW));
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = umma_overlap_launches ? 1 : 0;
  cudaLaunchKernelEx(&cfg, umma::k_conv_umma_mt<SUB, EPIW>, in, w, ls, sec, n_out, cin, cout, out, e, tmem_cols, na, nb, nsets);
}

// Configuration of k_conv_umma_mt for a layer: sub-tiles per super-tile come with the lists; accumulator
// sets, CTAs per SM and the two ring depths follow from tensor memory (512 columns per SM) and shared memory.
static int conv_umma_mt(const __half* in, const __half* w, const umma::Lists& ls, const umma::Second& sec, int n_out, int cin,
                        int cout, __half* out, const umma::Epi& e, int sub, int sm_count, cudaStream_t st) {
  if (sub != 1 && sub != 2 && sub != 4) return PCE_ERR_INVALID;
  if (sub * cout > 512) return PCE_ERR_UNSUPPORTED;
  static bool attr_set[64] = {};
  int dev = 0;
  PCE_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) return PCE_ERR_UNSUPPORTED;
  if (!attr_set[dev]) {
    const int cap = 227 * 1024;
    PCE_CUDA(cudaFuncSetAttribute(umma::k_conv_umma_mt<1, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, cap));
    PCE_CUDA(cudaFuncSetAttribute(umma::k_conv_umma_mt<2, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, cap));
    PCE_CUDA(cudaFuncSetAttribute(umma::k_conv_umma_mt<4, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, cap));
    attr_set[dev] = true;
  }
  // two CTAs per SM only for single sub-tiles with narrow accumulators (two sets of <= 128 columns each)
  const int ctas = (sub == 1 && 2 * cout <= 256) ? 2 : 1;
  int nsets = (2 * sub * cout * ctas <= 512) ? 2 : 1;
  if ((umma_force_nacc == 1 || umma_force_nacc == 2) && umma_force_nacc * sub * cout * ctas <= 512) nsets = umma_force_nacc;
  int tmem_cols = 32;
  while (tmem_cols < nsets * sub * cout) tmem_cols <<= 1;
  const size_t fixed = sizeof(umma::SharedCtlMt) + 1024 + 64;
  const size_t budget = static_cast<size_t>(227 * 1024) / ctas - fixed - (ctas > 1 ? 1024 : 0);
  const size_t b_bytes = static_cast<size_t>(cout) * 128;
  int nb = 3 * b_bytes * 3 <= budget ? 3 : 2;
  if (2 * b_bytes + 2 * umma::kABytes > budget) return PCE_ERR_UNSUPPORTED;
  // row slots per sub-tile; a third weight slot only where it does not cost a row slot per sub-tile
  int na = static_cast<int>((budget - nb * b_bytes) / umma::kABytes) / sub;
  if (nb == 3 && static_cast<int>((budget - 2 * b_bytes) / umma::kABytes) / sub > na) {
    nb = 2;
    na = static_cast<int>((budget - nb * b_bytes) / umma::kABytes) / sub;
  }
  if (na * sub > umma::kMaxA) na = umma::kMaxA / sub;
  if (umma_force_stages >= 2 && umma_force_stages <= na) na = umma_force_stages;
  if (na < 2) return PCE_ERR_UNSUPPORTED;
  const size_t smem = static_cast<size_t>(na) * sub * umma::kABytes + nb * b_bytes + fixed;
  const int n_tiles = div_up(n_out, umma::kTileM * sub);
  const int grid = n_tiles < sm_count * ctas ? n_tiles : sm_count * ctas;
  if (sub == 1)
    launch_umma_mt<1, 1>(grid, smem, st, in, w, ls, sec, n_out, cin, cout, out, e, tmem_cols, na, nb, nsets);
  else if (sub == 2)
    launch_umma_mt<2, 1>(grid, smem, st, in, w, ls, sec, n_out, cin, cout, out, e, tmem_cols, na, nb, nsets);
  else
    launch_umma_mt<4, 2>(grid, smem, st, in, w, ls, sec, n_out, cin, cout, out, e, tmem_cols, na, nb, nsets);
  PCE_LAUNCH_CHECK();
  return PCE_OK;
}

template <int NS, int SUB, bool PUSH, int SLOTS>
static void launch_umma(int grid, size_t smem, cudaStream_t st, const __half* in, const __half* w, const umma::Lists& ls,
                        const umma::Second& sec, int n_out, int cin, int cout, __half* out, const umma::Epi& e, int tmem_cols,
                        int nacc) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(32 * (4 * SUB + 5));
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  cfg.attrs = attr;
  if (umma_overlap_launches) {
    attr[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[cfg.numAttrs++].val.programmaticStreamSerializationAllowed = 1;
  }
  if (e.parts > 1) {
    attr[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
    attr[cfg.numAttrs].val.clusterDim.x = static_cast<unsigned>(e.parts);
    attr[cfg.numAttrs].val.clusterDim.y = 1;
    attr[cfg.numAttrs++].val.clusterDim.z = 1;
  }
  cudaLaunchKernelEx(&cfg, umma::k_conv_umma<NS, SUB, PUSH, SLOTS>, in, w, ls, sec, n_out, cin, cout, out, e, tmem_cols,
                     nacc);
}

// 1: maps with few tiles are split over several CTAs per tile, mid-size maps into equal shares of stages,
// when the caller asks for it (see conv_split_parts, conv_streamk_grid); 2: only the former; 0: never.
int umma_split_enabled = 1;

// Estimated ring stages per tile: min(kv, 16) offsets x K blocks, fewer where the map has fewer source rows than
// output rows (a transposed 2x2x2 layer has ONE pair per output row: its tiles list up to 8 offsets, each nearly
// empty, and splitting them only adds the partial sums; measured 16 -> 30 us on 159 tiles of 128 -> 128).
static int chain_estimate(int n_rows, int n_src, int cin, int kv) {
  long long offsets = kv < 16 ? kv : 16;
  if (n_src < n_rows) {
    const long long per_row = static_cast<long long>(kv) * n_src / n_rows;
    offsets = per_row < offsets ? (per_row > 1 ? per_row : 1) : offsets;
  }
  return static_cast<int>(offsets) * ((cin + 63) / 64);
}

// Input widths of k_conv_deep: whole K blocks, or a half block at the end (32 channels: one half block).
static bool deep_widths(int cin) { return cin >= 32 && cin % 32 == 0; }

// Layers of 32 input channels that k_conv_umma runs faster: it takes two offsets to a stage, which is half the
// stages, and up to four CTAs per SM, where a layer's set-up weighs.  Kernel only, us, k_conv_umma / k_conv_deep:
// * down and up a level (at most 8 offsets): 32->16 and 32->32 4.1 / 5.2 on 94 tiles, 5.6 / 7.0 on 326, 32->48 4.4 / 5.3 on 108, 42.7 / 46.7
//   on 5659 (on the way up 16.3 / 17.7 on 2415, 42.0 / 39.3 on 5434), 32->96 4.4 / 5.1 on 35 but 7.0 / 6.4 on 500; with one to three tiles per SM
//   also 32->64 (7.5 / 8.0 on 225) and on the way up 32->128 (6.2 / 7.4 on 199, 7.2 / 8.0 on 326).  (64->128 up: rooms 7.6 / 9.0 on 440, scans
//   9.0 / 8.4 on 426.)
// * other strided kernels that leave fewer rows: 32->32 6.8 / 8.8 on 279 tiles, 32->48 16.6 / 21.1 on 1781, but 7.7 / 7.2 on 104; 32->64
//   22.0 / 23.9 on 1820, but 20.9 / 18.8 on 233.
// * all others from five tiles per SM on: 32->32 15.7 / 17.1 on 938, 31.5 / 46.8 on 3750, but 32->48 16.5 / 14.5 on 798 (45.8 / 48.8 on 4322),
//   5x5x5 51.0 / 42.7 on 1489, 32->64 19.1 / 17.5 on 938.  Below that it depends on the cloud: 3x3x3 32->16 16.5 / 21.3 on 439 tiles of a
//   uniform one, 12.7 / 10.4 on 436 of a room.
static bool umma_faster(int n_out, int n_in, int cin, int cout, int kv, int sm_count) {
  const long long t = div_up(n_out, umma::kTileM), sms = sm_count;
  const bool mid = t > sms && t <= 3 * sms, many = t > 5 * sms;
  if (cin != 32) return false;
  if (kv <= 8) return cout <= 32 || (cout <= 48 && (n_in > n_out || t <= 16 * sms)) || (mid && cout <= (n_in < n_out ? 192 : 64));
  if (n_in > n_out) return (cout <= 48 && t > sms) || (cout <= 64 && many);
  return many && cout <= 32;
}

// Parts per tile of k_conv_deep (4, 2 or 1): as long as every part has an SM to itself and a chain worth cutting.  Kernel
// only, us, one / two / four parts: 256->256 on 24 tiles 39.3 / 27.6 / 20.4, on 60 tiles 38.2 / 27.5 / 34.4, on 94 tiles
// 31.2 / 34.1; 128->128 on 24 tiles 16.9 / 14.2 / 11.9, on 60 tiles 16.9 / 14.5 / 21.1; 64->64 on 24 tiles 10.3 / 10.2 / 9.2, on
// 60 tiles 10.4 / 10.4 / 16.8.  (Eight parts leave each a few stages: 256->256 on 24 tiles 30.5.)
// * Clusters of four find their SMs inside one GPC: 33 of them fit 148 SMs, not 37 (64->48 on 35 tiles 8.6 / - / 12.8; 5x5x5 64->160 on 33 tiles
//   - / 18.0 / 15.1).
// * At most 8 offsets (down and up a level): a row has few of them, one going up, so a part is a few stages.  None going up; two
//   going down need four K blocks, or three and narrow outputs (192->48 on 56 tiles 8.4 / 7.7 / 14.8, 256->64 on 46 8.4 / 8.2; 192->192 on 33
//   8.2 / 9.8).
// * More than 32 offsets: tiles at the end of the order have 125 where most have 20 to 50, and the layer lasts as long as
//   the longest chain, so cutting pays beyond an SM per part.  One K block (64->32): 67 tiles 17.7 / 11.7 / 18.7, 100 tiles 18.6 /
//   19.3.  More: 37 tiles 192->192 56 / 32.6 / 29.9, rooms of 82 tiles 96->128 49.5 / 36.7 / 34.3 and 256->48 68.4 / 44.2 / 36.2, a uniform
//   cloud of 88, where all tiles are alike, 256->96 94.7 / 86.9 / 81.1 (but four parts of a scan's short chains 256->64 on 84 tiles
//   23.7 / - / 29.9).  Above two thirds of the SMs it depends on the cloud: rooms 96->96 on 100 tiles 33.7 / 27.9, scans 160->96 on 101
//   20.1 / 22.1 and 256->256 on 103 60.7 / 51.4, uniform 128->128 on 107 51.4 / 57.5.
static int deep_split(int n_tiles, int n_out, int n_src, int cin, int cout, int kv, int sm_count) {
  if (!umma_split_enabled) return 1;
  const int chain = chain_estimate(n_out, n_src, cin, kv), kblocks = (cin + 63) / 64;
  const long long t = n_tiles;
  const bool two = 2 * t <= sm_count;
  if (chain < 16 || (kv <= 8 && n_src <= n_out)) return 1;
  if (40 * t <= 9 * sm_count) return 4;
  if (kv <= 8) return two && (chain >= 32 || (chain >= 24 && cout <= 64)) ? 2 : 1;
  if (kv <= 32) return two && chain >= 32 ? 2 : 1;
  if (kblocks == 1) return two ? 2 : 1;
  return 4 * t <= sm_count ? 4 : (3 * t <= 2 * sm_count ? 2 : 1);
}

// Parts per tile of k_conv_umma (8, 4, 2 or 1).  Layers with 16 input channels (shallow levels) are never split.
static int umma_split(int n_rows, int n_src, int cin, int cout, int kv, int sm_count) {
  if (!umma_split_enabled || n_rows < 1) return 1;
  const int cin_p = (cin + 15) / 16 * 16;
  if (cin_p == 16 || cin_p == 32) return 1;
  const int chain = chain_estimate(n_rows, n_src, cin, kv);
  const long long n_tiles = (static_cast<long long>(n_rows) + umma::kTileM - 1) / umma::kTileM;
  const long long sms = sm_count > 0 ? sm_count : 148;
  const long long slots = sms * (cout <= 128 ? 3 : 2);
  // Parts pay while their CTAs are resident at once and each keeps a few stages of a chain that costs 0.6 us a stage; eight
  // only where they still have about an SM each.  Whole -> split, us (3x3x3 on rooms, kernel only): 48->64 on 7.5 k rows 16.3 -> 8.5
  // (4 parts), on 25 k 17.6 -> 13.3 (2); 144->128 on 2.9 k rows 31.0 -> 11.8 (8), on 12 k 29.8 -> 16.0 (4), on 25 k 36.5 -> 25.0 (2);
  // 240->256 on 2.9 k rows 45.3 -> 19.8 (8), on 7.5 k 49.8 -> 23.1 (4), on 12 k 43.9 -> 31.1 (2); beyond the slots 128->256 on 23 k rows 38 -> 44.
  // The rows of a kernel of at most 8 offsets (down and up a level) have fewer of them than the estimate: twice the chain is
  // asked for.
  const int each = kv <= 8 ? 8 : 4;
  if (3 * n_tiles * 8 <= 4 * sms && chain >= each * 8) return 8;
  if (n_tiles * 4 <= slots && chain >= each * 4) return 4;
  if (n_tiles * 2 <= slots && chain >= each * 2) return 2;
  return 1;
}

// Parts per tile that conv_umma runs a layer with when its caller allows parts.
int conv_split_parts(int n_rows, int n_src, int cin, int cout, int kv, int sm_count) {
  if (n_rows < 1) return 1;
  if (deep_widths(cin) && !umma_faster(n_rows, n_src, cin, cout, kv, sm_count > 0 ? sm_count : 148))
    return deep_split(div_up(n_rows, umma::kTileM), n_rows, n_src, cin, cout, kv, sm_count > 0 ? sm_count : 148);
  return umma_split(n_rows, n_src, cin, cout, kv, sm_count);
}

// Maps of half a wave to one wave of tiles (tiles / CTA slots in (0.5, 1]) that umma_split leaves
// whole: CTAs take equal shares of the STAGES instead of whole tiles (stream-K), wherever the cuts fall, so
// every CTA slot works for the same time instead of some running a whole chain while others idle.  A tile
// that two or more CTAs worked on costs fp32 partial sums (written, then read by k_sum_cut_tiles), which is
// why it pays only for long chains on less than one wave.  Whole -> shares, us (kernel only, both kernels): 240->256 on 196 tiles
// of a scan 60.8 -> 50.6, on 235 of a room 56.1 -> 41.8; but 256->256 on 489 tiles (1.65 waves) 119 -> 136, 128->128 on 273 tiles 59 -> 58, and the
// 2x2x2 strided / transposed layers (chains of 8 offsets at most) 35-49 -> 56-65: those run whole.
// Returns the grid (= the CTA slots) or 0.
int conv_streamk_grid(int n_rows, int n_src, int cin, int cout, int kv, int sm_count) {
  if (!umma_split_enabled || umma_split_enabled == 2 || n_rows < 1) return 0;
  const int cin_p = (cin + 15) / 16 * 16;
  if (cin_p == 16 || cin_p == 32) return 0;
  if (umma_split(n_rows, n_src, cin, cout, kv, sm_count) > 1) return 0;
  const int chain = chain_estimate(n_rows, n_src, cin, kv);
  const long long n_tiles = (static_cast<long long>(n_rows) + umma::kTileM - 1) / umma::kTileM;
  const long long slots = static_cast<long long>(sm_count > 0 ? sm_count : 148) * (cout <= 128 ? 3 : 2);
  if (kv <= 8 || chain < 16 || 2 * n_tiles <= slots || n_tiles > slots) return 0;
  return static_cast<int>(slots);
}

// Scratch (bytes) that is enough for any split of a layer, 0 when it runs whole.  Parts need none: their bound is what
// callers of earlier versions sized by.
size_t conv_split_scratch_bytes(int n_rows, int n_src, int cin, int cout, int kv, int sm_count) {
  const int parts = conv_split_parts(n_rows, n_src, cin, cout, kv, sm_count);
  if (parts > 1) return static_cast<size_t>(parts) * n_rows * cout * sizeof(float);
  if (deep_widths(cin)) return 0;  // (k_conv_deep: shares three times as long leave little to balance)
  const int grid = conv_streamk_grid(n_rows, n_src, cin, cout, kv, sm_count);
  return grid > 0 ? static_cast<size_t>(grid) * 2 * umma::kTileM * cout * sizeof(float) : 0;
}

// The same where a split was measured faster; the framework's own callers ask this one.  Equal shares of stages repay
// their partial sums from chains of three K blocks on (whole -> shares, us: 144->128 on 235 tiles 37.9 -> 29.3, 176->192 on 196 39.8 -> 37.2,
// 240->256 53.6 -> 39.5; but 64->64 22 -> 27, 128->256 40 -> 57).
size_t conv_split_scratch_wanted(int n_rows, int n_src, int cin, int cout, int kv, int sm_count) {
  if (conv_split_parts(n_rows, n_src, cin, cout, kv, sm_count) > 1) return 0;  // (parts add up in shared memory)
  if (chain_estimate(n_rows, n_src, cin, kv) < 48) return 0;
  return conv_split_scratch_bytes(n_rows, n_src, cin, cout, kv, sm_count);
}

// cuTensorMapEncodeTiled, looked up once (the library does not link the driver's).
typedef CUresult (*EncodeTiled)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static EncodeTiled encode_tiled() {
  static EncodeTiled fn = nullptr;
  EncodeTiled f = __atomic_load_n(&fn, __ATOMIC_RELAXED);
  if (!f) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult found;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &found) != cudaSuccess || found != cudaDriverEntryPointSuccess)
      return nullptr;
    f = reinterpret_cast<EncodeTiled>(p);
    __atomic_store_n(&fn, f, __ATOMIC_RELAXED);
  }
  return f;
}

// Rows of `width` fp16 values, `pitch` apart, as boxes of one row x `box` channels (64: 128-byte swizzle, 32: 64-byte).
static bool row_map(CUtensorMap* map, const void* base, long long rows, int width, int pitch, int box) {
  const EncodeTiled encode = encode_tiled();
  if (!encode || rows < 1) return false;
  const cuuint64_t dim[2] = {static_cast<cuuint64_t>(width), static_cast<cuuint64_t>(rows)}, stride[1] = {static_cast<cuuint64_t>(pitch) * 2};
  const cuuint32_t boxes[2] = {static_cast<cuuint32_t>(box), 1}, step[2] = {1, 1};
  return encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void*>(base), dim, stride, boxes, step, CU_TENSOR_MAP_INTERLEAVE_NONE,
                box == 64 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

typedef void (*DeepKernel)(const umma::DeepMaps, const __half*, const umma::Lists, const umma::Second, int, int, int, __half*, const umma::Epi, int, int);
static DeepKernel deep_kernel(bool half, int ring) {
  static const DeepKernel table[2][6] = {
      {umma::k_conv_deep<false, 4>, umma::k_conv_deep<false, 5>, umma::k_conv_deep<false, 6>, umma::k_conv_deep<false, 7>,
       umma::k_conv_deep<false, 8>, umma::k_conv_deep<false, 9>},
      {umma::k_conv_deep<true, 4>, umma::k_conv_deep<true, 5>, umma::k_conv_deep<true, 6>, umma::k_conv_deep<true, 7>,
       umma::k_conv_deep<true, 8>, umma::k_conv_deep<true, 9>}};
  return table[half ? 1 : 0][ring - 4];
}

// tiles == nullptr: the dense rows x matrix product (every row fetches itself, one offset).
static int conv_umma_impl(const void* in, int n_in, const void* wpacked, int kv, const pce_tile_lists* tiles, int n_out,
                          int cin, int cout, void* out, const pce_epilogue* ep, cudaStream_t st, bool kb64_slice);

int conv_umma(const void* in, int n_in, const void* wpacked, int kv, const pce_tile_lists* tiles, int n_out, int cin,
              int cout, void* out, const pce_epilogue* ep, cudaStream_t st) {
  return conv_umma_impl(in, n_in, wpacked, kv, tiles, n_out, cin, cout, out, ep, st, false);
}

// The same for weights that are a SLICE of a larger packed buffer (one offset's 64-channel blocks): there is no
// second image behind them, so the layer runs with 64-channel K blocks whatever its width.
int conv_umma_kb64(const void* in, int n_in, const void* wpacked, int kv, const pce_tile_lists* tiles, int n_out, int cin,
                   int cout, void* out, const pce_epilogue* ep, cudaStream_t st) {
  return conv_umma_impl(in, n_in, wpacked, kv, tiles, n_out, cin, cout, out, ep, st, true);
}

// `split`: the caller allows several CTAs per tile.
static int conv_deep(const umma::DeepMaps& maps, const __half* w, const umma::Lists& ls, const umma::Second& sec, int n_in, int n_out, int cin,
                     int cout, int kv, __half* out, umma::Epi e, bool half, bool split, int dev, int sm_count, cudaStream_t st) {
  const size_t stage = static_cast<size_t>(umma::kABytes) + static_cast<size_t>(cout) * 128;
  const size_t rest = sizeof(umma::DeepCtl) + 1024 + 64 + 2 * sizeof(float) * cout;
  const int ring = std::min<int>(umma::kDeepMaxRing, static_cast<int>((227 * 1024 - rest) / stage));
  static bool attr_set[64][2][umma::kDeepMaxRing + 1] = {};  // (a variant is loaded when it is first wanted)
  if (!attr_set[dev][half][ring]) {
    PCE_CUDA(cudaFuncSetAttribute(reinterpret_cast<const void*>(deep_kernel(half, ring)), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  227 * 1024));
    attr_set[dev][half][ring] = true;
  }
  const int nacc = cout <= 128 ? 4 : 2;
  int cols = 32;
  while (cols < nacc * cout) cols <<= 1;
  const int n_tiles = div_up(n_out, umma::kTileM);
  const int parts = split && !ls.tall ? deep_split(n_tiles, n_out, n_in, cin, cout, kv, sm_count) : 1;
  e.parts = parts;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(parts > 1 ? n_tiles * parts : std::min((n_tiles + ls.tall) >> ls.tall, sm_count));
  cfg.blockDim = dim3(umma::deep_threads(ring));
  cfg.dynamicSmemBytes = ring * stage + rest;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  cfg.attrs = attr;
  if (umma_overlap_launches) {
    attr[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[cfg.numAttrs++].val.programmaticStreamSerializationAllowed = 1;
  }
  if (parts > 1) {
    attr[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
    attr[cfg.numAttrs].val.clusterDim.x = static_cast<unsigned>(parts);
    attr[cfg.numAttrs].val.clusterDim.y = 1;
    attr[cfg.numAttrs++].val.clusterDim.z = 1;
  }
  PCE_CUDA(cudaLaunchKernelEx(&cfg, deep_kernel(half, ring), maps, w, ls, sec, n_out, cin, cout, out, e, cols, nacc));
  PCE_LAUNCH_CHECK();
  return PCE_OK;
}

static int conv_umma_impl(const void* in, int n_in, const void* wpacked, int kv, const pce_tile_lists* tiles, int n_out,
                          int cin, int cout, void* out, const pce_epilogue* ep, cudaStream_t st, bool kb64_slice) {
  umma::Epi e{nullptr, nullptr, nullptr, PCE_ACT_NONE, 0.f, {nullptr, nullptr}, {nullptr, nullptr}, cin, cout};
  if (ep) {
    e = umma::Epi{ep->scale, ep->shift, static_cast<const __half*>(ep->residual), ep->act, ep->slope,
                  {ep->push_slot[0], ep->push_slot[1]},
                  {static_cast<__half*>(ep->push_base[0]), static_cast<__half*>(ep->push_base[1])},
                  ep->in_ld > 0 ? ep->in_ld : cin, ep->out_ld > 0 ? ep->out_ld : cout};
    // rows stay 16-byte aligned: the pitch is a multiple of 8 halves and covers the channels
    if (e.ld_in < cin || e.ld_out < cout || (e.ld_in & 7) || (e.ld_out & 7)) return PCE_ERR_INVALID;
    if (off16(ep->residual) || off16(ep->extra_feats, ep->extra_packed_weights)) return PCE_ERR_INVALID;
    for (int s = 0; s < 2; ++s) {
      if (e.push_slot[s] && (!e.push_base[s] || (reinterpret_cast<uintptr_t>(e.push_base[s]) & 15))) return PCE_ERR_INVALID;
      if (!e.push_slot[s]) e.push_base[s] = nullptr;
    }
  }
  umma::Lists ls{nullptr, nullptr, nullptr, nullptr, 0, nullptr, nullptr, 0, 1, 0};
  int slots = 1;
  umma::Second sec{nullptr, nullptr, nullptr, 0};
  int sub = umma_force_sub == 1 || umma_force_sub == 2 ? umma_force_sub : 1;
  if (tiles) {
    ls = umma::Lists{tiles->order, tiles->tile_ptr, tiles->stage_kp, tiles->stage_nbr, tiles->identity_stage ? 1 : 0, nullptr, nullptr,
                     (tiles->settled && umma_overlap_launches == 1) ? 1 : 0, 1, 0};
    slots = tiles->slots > 1 ? tiles->slots : 1;
    if (slots != 1) {
      // several offsets per stage: the lists must match the layer's width, and the packed weights carry
      // the per-offset [cout][cin] images behind the per-offset blocks
      if ((slots != 2 && slots != 4) || cin * slots != 64) return PCE_ERR_INVALID;
      ls.wslots = static_cast<const __half*>(wpacked) + static_cast<size_t>(kv) * cout * 64;
    }
    if (tiles->tile_rows != 128 && tiles->tile_rows != 256 && tiles->tile_rows != 512) return PCE_ERR_INVALID;
    sub = tiles->tile_rows / 128;  // the lists fix the tile height
  }
  if (sub * cout > 512) return PCE_ERR_UNSUPPORTED;
  if (sub > 2 && (slots != 1 || !tiles)) return PCE_ERR_UNSUPPORTED;
  if (ep && ep->extra_feats) {
    // the second operand rides on the identity stage of the tile lists
    if (!ls.identity || !ep->extra_packed_weights || ep->extra_c < 16 || ep->extra_c % 16) return PCE_ERR_UNSUPPORTED;
    sec = umma::Second{static_cast<const __half*>(ep->extra_feats), static_cast<const __half*>(ep->extra_packed_weights), nullptr,
                       ep->extra_c};
  }
  const size_t fixed = sizeof(umma::SharedCtl) + 1024 + 64 + 2 * sizeof(float) * cout;  // (+ staged scale / shift)
  const size_t stage = static_cast<size_t>(umma::kABytes) * sub + static_cast<size_t>(cout) * 128;
  static int sm_count[64] = {};
  // registers per thread by kernel variant (plain, push, 2 slots, 4 slots) and sub-tile count, in
  // allocation units of 8; read back from the compiled kernels at set-up
  static int regs_per_thread[4][2] = {{72, 72}, {80, 80}, {80, 80}, {96, 88}};
  int dev = 0;
  PCE_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) return PCE_ERR_UNSUPPORTED;
  if (sm_count[dev] == 0) {
    const int cap = 227 * 1024;
#define PCE_SET_SMEM(NS, SB) \
  PCE_CUDA(cudaFuncSetAttribute(umma::k_conv_umma<NS, SB, false, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, cap)); \
  PCE_CUDA(cudaFuncSetAttribute(umma::k_conv_umma<NS, SB, true, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, cap));  \
  PCE_CUDA(cudaFuncSetAttribute(umma::k_conv_umma<NS, SB, false, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, cap)); \
  PCE_CUDA(cudaFuncSetAttribute(umma::k_conv_umma<NS, SB, false, 4>, cudaFuncAttributeMaxDynamicSharedMemorySize, cap))
    PCE_SET_SMEM(4, 1);
    PCE_SET_SMEM(3, 1);
    PCE_SET_SMEM(2, 1);
    PCE_SET_SMEM(4, 2);
    PCE_SET_SMEM(3, 2);
    PCE_SET_SMEM(2, 2);
#undef PCE_SET_SMEM
    cudaFuncAttributes fa;
#define PCE_REGS(V, SB, KERNEL) \
  if (cudaFuncGetAttributes(&fa, KERNEL) == cudaSuccess && fa.numRegs > 0) regs_per_thread[V][SB - 1] = (fa.numRegs + 7) / 8 * 8
    PCE_REGS(0, 1, (umma::k_conv_umma<2, 1, false, 1>));
    PCE_REGS(0, 2, (umma::k_conv_umma<2, 2, false, 1>));
    PCE_REGS(1, 1, (umma::k_conv_umma<2, 1, true, 1>));
    PCE_REGS(1, 2, (umma::k_conv_umma<2, 2, true, 1>));
    PCE_REGS(2, 1, (umma::k_conv_umma<2, 1, false, 2>));
    PCE_REGS(2, 2, (umma::k_conv_umma<2, 2, false, 2>));
    PCE_REGS(3, 1, (umma::k_conv_umma<2, 1, false, 4>));
    PCE_REGS(3, 2, (umma::k_conv_umma<2, 2, false, 4>));
#undef PCE_REGS
    int n = 0;
    PCE_CUDA(cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev));
    sm_count[dev] = n > 0 ? n : 1;
  }
  {
    const bool push_any = e.push_slot[0] || e.push_slot[1];
    if (tiles && slots == 1 && !push_any && (umma_multi_tile || sub == 4))
      return conv_umma_mt(static_cast<const __half*>(in), static_cast<const __half*>(wpacked), ls, sec, n_out, cin, cout,
                          static_cast<__half*>(out), e, sub, sm_count[dev], st);
    if (sub > 2) return PCE_ERR_UNSUPPORTED;  // 512-row super-tiles exist for k_conv_umma_mt only
  }
  // One CTA per SM wherever its producers can take the layer (k_conv_deep); the tuning hooks below are k_conv_umma's.
  const bool pairs = slots == 2;  // 32 input channels: a half block per offset there, two offsets to a stage below
  const bool deep_half = !kb64_slice && cin % 64 == 32;  // (a slice of a packed buffer has no second image behind it)
  const bool packed = pairs && umma_faster(n_out, n_in, cin, cout, kv, sm_count[dev]);
  if (!packed && (slots == 1 ? sub == 1 : pairs) && !(e.push_slot[0] || e.push_slot[1]) && deep_widths(cin) && (cin % 64 == 0 || deep_half) && !off16(in) &&
      !off16(ls.stage_nbr) && !umma_force_stages && !umma_force_nacc) {
    umma::Lists dl = ls;
    umma::Second ds = sec;
    dl.entries = pairs ? 2 : 1;
    dl.tall = sub == 2 ? 1 : 0;
    if (deep_half) {
      dl.wtail = reinterpret_cast<const __half*>(static_cast<const char*>(wpacked) + kb64_image_bytes(kv, cin, cout));
      if (ds.in2 && ds.cin2 % 64 == 32)
        ds.wtail = reinterpret_cast<const __half*>(reinterpret_cast<const char*>(ds.w2) + kb64_image_bytes(1, ds.cin2, cout));
    }
    umma::DeepMaps maps;
    bool mapped = row_map(&maps.in, in, n_in, cin, e.ld_in, 64) && (!deep_half || row_map(&maps.in32, in, n_in, cin, e.ld_in, 32));
    if (ds.in2)
      mapped = mapped && row_map(&maps.sec, ds.in2, n_out, ds.cin2, ds.cin2, 64) &&
               (!ds.wtail || row_map(&maps.sec32, ds.in2, n_out, ds.cin2, ds.cin2, 32));
    if (mapped)
      return conv_deep(maps, static_cast<const __half*>(wpacked), dl, ds, n_in, n_out, cin, cout, kv, static_cast<__half*>(out), e,
                       deep_half, tiles && ep && (ep->split || ep->split_scratch), dev, sm_count[dev], st);
  }
  // Configuration = (ring depth, accumulator sets).  What the kernel needs most is row gathers in
  // flight, i.e. stages resident per SM = resident CTAs x ring depth; the CTAs per SM are bounded by
  // shared memory, by the 512 tensor-memory columns and by the register file.  Measured on LiDAR
  // layers (486k / 297k / 149k rows): at an equal stage count more CTAs win (C=96: 3 CTAs x 2 stages
  // with one accumulator set 146 us, 2 x 3 with two sets 159 us; C=128: 115 vs 122 us), and at equal
  // CTAs two accumulator sets win (the epilogue of a tile then overlaps the next tile's MMAs).
  const int threads = 32 * (4 * sub + 5);
  const bool push = e.push_slot[0] || e.push_slot[1];
  if (push && slots != 1) return PCE_ERR_UNSUPPORTED;  // the halo push has no several-offsets-per-stage variant
  const int variant = push ? 1 : (slots == 2 ? 2 : (slots == 4 ? 3 : 0));
  const int by_regs = 65536 / (threads * regs_per_thread[variant][sub - 1]);
  auto tmem_for = [&](int sets) {
    int cols = 32;
    while (cols < sets * sub * cout) cols <<= 1;
    return cols;
  };
  auto ctas_for = [&](int n, int sets) {
    if (sets * sub * cout > 512) return 0;
    int c = static_cast<int>((227 * 1024) / (n * stage + fixed + 1024));
    if (c > 512 / tmem_for(sets)) c = 512 / tmem_for(sets);
    if (c > by_regs) c = by_regs;
    return c > 4 ? 4 : c;
  };
  int ns = 2, nacc = 1, per_sm = 0;
  for (int n = 4; n >= 2; --n) {
    for (int sets = 2; sets >= 1; --sets) {
      const int c = ctas_for(n, sets);
      const bool better = c * n > per_sm * ns || (c * n == per_sm * ns && c > per_sm);
      if (c > 0 && (per_sm == 0 || better)) {
        ns = n;
        nacc = sets;
        per_sm = c;
      }
    }
  }
  if (umma_force_stages >= 2 && umma_force_stages <= 4) ns = umma_force_stages;
  if ((umma_force_nacc == 1 || umma_force_nacc == 2) && umma_force_nacc * sub * cout <= 512) nacc = umma_force_nacc;
  per_sm = ctas_for(ns, nacc);
  const int tmem_cols = tmem_for(nacc);
  if (per_sm < 1) per_sm = 1;
  const size_t smem = ns * stage + fixed;
  if (smem > 227 * 1024) return PCE_ERR_UNSUPPORTED;
  const int n_tiles = div_up(n_out, umma::kTileM * sub);
  int grid = n_tiles < sm_count[dev] * per_sm ? n_tiles : sm_count[dev] * per_sm;
  // few tiles, long stage chains: several CTAs per tile, or shares of stages with partial sums in the caller's scratch
  int parts = 1;
  bool streamk = false;
  const bool scratch = ep && ep->split_scratch && (reinterpret_cast<uintptr_t>(ep->split_scratch) & 15) == 0;
  if (tiles && sub == 1 && slots == 1 && !push && ep && (ep->split || scratch)) {
    parts = umma_split(n_out, n_in, cin, cout, kv, sm_count[dev]);
    if (parts > 1) {
      grid = n_tiles * parts;
      e.parts = parts;
    } else if (scratch) {
      const int g = conv_streamk_grid(n_out, n_in, cin, cout, kv, sm_count[dev]);
      if (g > 0 && g <= sm_count[dev] * per_sm &&
          static_cast<size_t>(g) * 2 * umma::kTileM * cout * sizeof(float) <= ep->split_scratch_bytes) {
        grid = g;
        streamk = true;
        e.partial = static_cast<float*>(ep->split_scratch);
        e.streamk = 1;
      }
    }
  }
  const __half* in_h = static_cast<const __half*>(in);
  const __half* w_h = static_cast<const __half*>(wpacked);
  __half* out_h = static_cast<__half*>(out);
#define PCE_GO(NS, SB)                                                                                              \
  do {                                                                                                              \
    if (push)                                                                                                         \
      launch_umma<NS, SB, true, 1>(grid, smem, st, in_h, w_h, ls, sec, n_out, cin, cout, out_h, e, tmem_cols, nacc);  \
    else if (slots == 2)                                                                                              \
      launch_umma<NS, SB, false, 2>(grid, smem, st, in_h, w_h, ls, sec, n_out, cin, cout, out_h, e, tmem_cols, nacc); \
    else if (slots == 4)                                                                                              \
      launch_umma<NS, SB, false, 4>(grid, smem, st, in_h, w_h, ls, sec, n_out, cin, cout, out_h, e, tmem_cols, nacc); \
    else                                                                                                              \
      launch_umma<NS, SB, false, 1>(grid, smem, st, in_h, w_h, ls, sec, n_out, cin, cout, out_h, e, tmem_cols, nacc); \
  } while (0)
  if (sub == 1) {
    if (ns == 4) PCE_GO(4, 1); else if (ns == 3) PCE_GO(3, 1); else PCE_GO(2, 1);
  } else {
    if (ns == 4) PCE_GO(4, 2); else if (ns == 3) PCE_GO(3, 2); else PCE_GO(2, 2);
  }
#undef PCE_GO
  PCE_LAUNCH_CHECK();
  if (streamk) {
    // the second kernel of a stream-K layer is set up on the SMs while the convolution's last CTAs drain
    // (programmatic dependent launch; it waits for that grid before it reads a partial sum)
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.blockDim = dim3(256);
    cfg.stream = st;
    cfg.attrs = attr;
    cfg.numAttrs = umma_overlap_launches ? 1 : 0;
    cfg.gridDim = dim3(div_up(umma::kTileM * (cout >> 3), 256), n_tiles);
    const float* partial = e.partial;
    const int* tile_ptr = ls.tile_ptr;
    const int* order = ls.order;
    cudaLaunchKernelEx(&cfg, umma::k_sum_cut_tiles, partial, tile_ptr, order, n_tiles, grid, n_out, cout, out_h, e);
    PCE_LAUNCH_CHECK();
  }
  return PCE_OK;
}

int umma_where_fetch(int* host4) {
  PCE_CUDA(cudaMemcpyFromSymbol(host4, g_umma_where, 4 * sizeof(int)));
  int z[4] = {0, 0, 0, 0};
  PCE_CUDA(cudaMemcpyToSymbol(g_umma_where, z, 4 * sizeof(int)));
  return PCE_OK;
}

int umma_status_fetch(int* host_status, bool reset) {
  int v = 0;
  PCE_CUDA(cudaMemcpyFromSymbol(&v, g_umma_status, sizeof(int)));
  if (reset && v != 0) {
    int z = 0;
    PCE_CUDA(cudaMemcpyToSymbol(g_umma_status, &z, sizeof(int)));
  }
  *host_status = v;
  return PCE_OK;
}

}  // namespace pce

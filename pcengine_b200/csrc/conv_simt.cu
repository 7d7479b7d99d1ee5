// CUDA-core fused gather-matmul-scatter (output stationary) for narrow or odd
// channel counts, the dense rows x matrix product, and the stand-alone
// scale/shift/activation pass.  A group of G threads owns one output row; each
// thread keeps four fp32 accumulators (four consecutive output channels),
// walks the row's neighbour list once and stores the row once with the fused
// epilogue.  Weights are read through the read-only path and stay L1/L2
// resident.  Role of the reference's CUDA-core fetch-on-demand kernels
// (ref: backend/spconv.cuh:427-735,832-935,1162-1250) without their atomics.
#include <algorithm>

#include "common.cuh"

namespace pce {

struct EpiDev {
  const float* scale;
  const float* shift;
  const void* residual;
  int act;
  float slope;
};

static EpiDev to_dev(const pce_epilogue* ep) {
  EpiDev e{nullptr, nullptr, nullptr, PCE_ACT_NONE, 0.f};
  if (ep) {
    e.scale = ep->scale;
    e.shift = ep->shift;
    e.residual = ep->residual;
    e.act = ep->act;
    e.slope = ep->slope;
  }
  return e;
}

__device__ __forceinline__ float to_f(float v) { return v; }
__device__ __forceinline__ float to_f(__half v) { return __half2float(v); }
template <typename T>
__device__ __forceinline__ T from_f(float v);
template <>
__device__ __forceinline__ float from_f<float>(float v) {
  return v;
}
template <>
__device__ __forceinline__ __half from_f<__half>(float v) {
  return __float2half_rn(v);
}

__device__ __forceinline__ float apply_act(float v, int act, float slope) {
  if (act == PCE_ACT_RELU) return v > 0.f ? v : 0.f;
  if (act == PCE_ACT_LEAKY) return v > 0.f ? v : v * slope;
  return v;
}

template <typename T>
__device__ __forceinline__ void store_row4(T* out, const EpiDev& ep, size_t row, int cout, int co0,
                                           const float (&acc)[4]) {
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    int c = co0 + j;
    if (c < cout) {
      float v = acc[j];
      if (ep.scale) v *= __ldg(ep.scale + c);
      if (ep.shift) v += __ldg(ep.shift + c);
      if (ep.residual) v += to_f(static_cast<const T*>(ep.residual)[row * cout + c]);
      out[row * cout + c] = from_f<T>(apply_act(v, ep.act, ep.slope));
    }
  }
}

// acc[0..3] += x_row[0..cin) . W[:, co0..co0+3]
template <typename T, bool VEC>
__device__ __forceinline__ void row_times_w(const T* __restrict__ xrow, const T* __restrict__ wk, int cin, int cout,
                                            int co0, float (&acc)[4]);

template <>
__device__ __forceinline__ void row_times_w<float, true>(const float* __restrict__ xrow, const float* __restrict__ wk,
                                                         int cin, int cout, int co0, float (&acc)[4]) {
  for (int ci = 0; ci < cin; ci += 4) {
    const float4 x = __ldg(reinterpret_cast<const float4*>(xrow + ci));
    const float xs[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      const float4 w = __ldg(reinterpret_cast<const float4*>(wk + static_cast<size_t>(ci + t) * cout + co0));
      acc[0] = fmaf(xs[t], w.x, acc[0]);
      acc[1] = fmaf(xs[t], w.y, acc[1]);
      acc[2] = fmaf(xs[t], w.z, acc[2]);
      acc[3] = fmaf(xs[t], w.w, acc[3]);
    }
  }
}

template <>
__device__ __forceinline__ void row_times_w<__half, true>(const __half* __restrict__ xrow,
                                                          const __half* __restrict__ wk, int cin, int cout, int co0,
                                                          float (&acc)[4]) {
  for (int ci = 0; ci < cin; ci += 8) {
    const uint4 xr = __ldg(reinterpret_cast<const uint4*>(xrow + ci));
    const __half2* xh = reinterpret_cast<const __half2*>(&xr);
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      const float2 xf = __half22float2(xh[t]);
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const float xv = u ? xf.y : xf.x;
        const uint2 wr = __ldg(reinterpret_cast<const uint2*>(wk + static_cast<size_t>(ci + 2 * t + u) * cout + co0));
        const float2 w01 = __half22float2(*reinterpret_cast<const __half2*>(&wr.x));
        const float2 w23 = __half22float2(*reinterpret_cast<const __half2*>(&wr.y));
        acc[0] = fmaf(xv, w01.x, acc[0]);
        acc[1] = fmaf(xv, w01.y, acc[1]);
        acc[2] = fmaf(xv, w23.x, acc[2]);
        acc[3] = fmaf(xv, w23.y, acc[3]);
      }
    }
  }
}

template <typename T>
__device__ __forceinline__ void row_times_w_scalar(const T* __restrict__ xrow, const T* __restrict__ wk, int cin,
                                                   int cout, int co0, float (&acc)[4]) {
  for (int ci = 0; ci < cin; ++ci) {
    const float xv = to_f(xrow[ci]);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (co0 + j < cout) acc[j] = fmaf(xv, to_f(wk[static_cast<size_t>(ci) * cout + co0 + j]), acc[j]);
    }
  }
}

template <>
__device__ __forceinline__ void row_times_w<float, false>(const float* __restrict__ xrow,
                                                          const float* __restrict__ wk, int cin, int cout, int co0,
                                                          float (&acc)[4]) {
  row_times_w_scalar<float>(xrow, wk, cin, cout, co0, acc);
}
template <>
__device__ __forceinline__ void row_times_w<__half, false>(const __half* __restrict__ xrow,
                                                           const __half* __restrict__ wk, int cin, int cout, int co0,
                                                           float (&acc)[4]) {
  row_times_w_scalar<__half>(xrow, wk, cin, cout, co0, acc);
}

// IDENT: every row has exactly the pair (row, kp 0, row) -- the dense product.
template <typename T, bool VEC, bool IDENT>
__global__ void __launch_bounds__(256)
    k_conv_simt(const T* __restrict__ in, const T* __restrict__ w, const uint32_t* __restrict__ mask,
                const int* __restrict__ rowptr, const int* __restrict__ nbr, int n_out, int cin, int cout, int kv,
                T* __restrict__ out, EpiDev ep, int g_threads) {
  const int rows_per_block = blockDim.x / g_threads;
  const int row = blockIdx.x * rows_per_block + threadIdx.x / g_threads;
  const int g = threadIdx.x % g_threads;
  if (row >= n_out) return;
  const int words = (kv + 31) / 32;
  const size_t wslab = static_cast<size_t>(cin) * cout;
  for (int co0 = g * 4; co0 < cout; co0 += g_threads * 4) {
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
    if (IDENT) {
      row_times_w<T, VEC>(in + static_cast<size_t>(row) * cin, w, cin, cout, co0, acc);
    } else {
      int p = __ldg(rowptr + row);
      for (int wd = 0; wd < words; ++wd) {
        uint32_t m = __ldg(mask + static_cast<size_t>(row) * words + wd);
        while (m) {
          const int kp = wd * 32 + __ffs(m) - 1;
          m &= m - 1;
          const int nid = __ldg(nbr + p);
          ++p;
          row_times_w<T, VEC>(in + static_cast<size_t>(nid) * cin, w + kp * wslab, cin, cout, co0, acc);
        }
      }
    }
    store_row4<T>(out, ep, static_cast<size_t>(row), cout, co0, acc);
  }
}

// Per-channel affine (+ residual, activation) over a dense row-major matrix, taken as one long run of 16-byte pieces:
// bound by memory alone (it moves each value in once and out once).  A block first puts the channels' scale and shift
// into shared memory -- as given, or from the statistics and parameters of an eval-mode BatchNorm, which then needs no
// kernels of its own to fold them -- and every thread takes kPieces pieces a grid apart, all loads in flight before the
// first use.  The channel of a piece is carried along (one addition per step) instead of divided out.
struct NormSrc {
  const void* mean;
  const void* var;
  const void* gamma;  // may be nullptr
  const void* beta;   // may be nullptr
  float eps;
  int half;  // the four are fp16 (else fp32)
};

__device__ __forceinline__ float param_at(const void* p, int half, int c) {
  return half ? __half2float(static_cast<const __half*>(p)[c]) : static_cast<const float*>(p)[c];
}

// MODE 0: the grid's stride is a whole number of rows, so a thread meets the same channels in every piece and keeps
// their constants in registers (read per piece, they are 32-byte-strided shared-memory reads that take as long as the
// memory traffic); 1: pieces lie within a row; 2: a piece may span rows (widths that are no multiple of a piece).
// RES: with a residual.  Both kept apart so that the pass without one needs 64 registers and an SM holds four blocks of it: with
// the residual's pieces in every variant it took 111, two blocks, and 240 k x 96 fp16 values (92 MB) 22.1 us; now 14.2 (6.5 TB/s, much of it L2).
template <typename T, int MODE, bool RES>
__global__ void __launch_bounds__(256, RES ? 3 : 4) k_scale_shift_act(const T* __restrict__ x, long long total, int c, T* __restrict__ y, EpiDev ep,
                                                         NormSrc norm, int staged) {
  constexpr int kVec = 16 / static_cast<int>(sizeof(T));
  constexpr int kPieces = 4;
  extern __shared__ __align__(16) float affine[];  // [2][c] when staged
  const float* scale = ep.scale;
  const float* shift = ep.shift;
  if (staged) {
    for (int ch = threadIdx.x; ch < c; ch += blockDim.x) {
      float s = 1.f, t = 0.f;
      if (norm.mean) {
        s = (norm.gamma ? param_at(norm.gamma, norm.half, ch) : 1.f) / sqrtf(param_at(norm.var, norm.half, ch) + norm.eps);
        t = (norm.beta ? param_at(norm.beta, norm.half, ch) : 0.f) - param_at(norm.mean, norm.half, ch) * s;
      } else {
        if (ep.scale) s = ep.scale[ch];
        if (ep.shift) t = ep.shift[ch];
      }
      affine[ch] = s;
      affine[c + ch] = t;
    }
    __syncthreads();
    scale = affine;
    shift = affine + c;
  }
  const long long pieces = total / kVec;
  const long long stride = static_cast<long long>(gridDim.x) * blockDim.x;
  const long long i0 = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  auto one = [&](float v, int ch, float r) {
    if (scale) v *= scale[ch];
    if (shift) v += shift[ch];
    return apply_act(v + r, ep.act, ep.slope);
  };
  int ch = static_cast<int>(i0 * kVec % c);
  float s_mine[kVec], t_mine[kVec];
  if (MODE == 0) {
#pragma unroll
    for (int u = 0; u < kVec; ++u) {
      s_mine[u] = scale[ch + u];
      t_mine[u] = shift[ch + u];
    }
  }
  const int step = static_cast<int>(stride * kVec % c);
  for (long long i = i0; i < pieces; i += kPieces * stride) {
    uint4 v[kPieces], r[RES ? kPieces : 1];
#pragma unroll
    for (int q = 0; q < kPieces; ++q) {
      const long long at = i + q * stride;
      if (at < pieces) {
        v[q] = *reinterpret_cast<const uint4*>(x + at * kVec);
        if (RES) r[RES ? q : 0] = *reinterpret_cast<const uint4*>(static_cast<const T*>(ep.residual) + at * kVec);
      }
    }
#pragma unroll
    for (int q = 0; q < kPieces; ++q) {
      const long long at = i + q * stride;
      if (at < pieces) {
        const T* pv = reinterpret_cast<const T*>(&v[q]);
        const T* pr = reinterpret_cast<const T*>(&r[RES ? q : 0]);
        alignas(16) T o[kVec];
        if (MODE == 0) {
#pragma unroll
          for (int u = 0; u < kVec; ++u)
            o[u] = from_f<T>(apply_act(to_f(pv[u]) * s_mine[u] + t_mine[u] + (RES ? to_f(pr[u]) : 0.f), ep.act, ep.slope));
        } else {
          int cc = ch;
#pragma unroll
          for (int u = 0; u < kVec; ++u) {
            o[u] = from_f<T>(one(to_f(pv[u]), cc, RES ? to_f(pr[u]) : 0.f));
            ++cc;
            if (MODE == 2 && cc == c) cc = 0;
          }
        }
        *reinterpret_cast<uint4*>(y + at * kVec) = *reinterpret_cast<const uint4*>(o);
      }
      if (MODE != 0) {
        ch += step;
        if (ch >= c) ch -= c;
      }
    }
  }
  const long long e = pieces * kVec + i0;  // the last, incomplete piece
  if (e < total)
    y[e] = from_f<T>(one(to_f(x[e]), static_cast<int>(e % c), RES ? to_f(static_cast<const T*>(ep.residual)[e]) : 0.f));
}

// Matrices that do not start on a 16-byte boundary.
template <typename T>
__global__ void k_scale_shift_act_unaligned(const T* __restrict__ x, long long total, int c, T* __restrict__ y, EpiDev ep) {
  long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  for (; i < total; i += static_cast<long long>(gridDim.x) * blockDim.x) {
    int ch = static_cast<int>(i % c);
    float v = to_f(x[i]);
    if (ep.scale) v *= __ldg(ep.scale + ch);
    if (ep.shift) v += __ldg(ep.shift + ch);
    if (ep.residual) v += to_f(static_cast<const T*>(ep.residual)[i]);
    y[i] = from_f<T>(apply_act(v, ep.act, ep.slope));
  }
}

template <typename T>
static int launch_affine(const void* x, long long total, int c, void* y, const EpiDev& e, const NormSrc& norm, cudaStream_t st) {
  constexpr int kVec = 16 / static_cast<int>(sizeof(T));
  const T* x_t = static_cast<const T*>(x);
  T* y_t = static_cast<T*>(y);
  const bool aligned = ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(y) | reinterpret_cast<uintptr_t>(e.residual)) & 15) == 0;
  if (!aligned) {
    if (norm.mean) return PCE_ERR_UNSUPPORTED;
    k_scale_shift_act_unaligned<T><<<static_cast<int>(std::min<long long>((total + 255) / 256, 148ll * 16)), 256, 0, st>>>(x_t, total, c, y_t, e);
    PCE_LAUNCH_CHECK();
    return PCE_OK;
  }
  const size_t smem = sizeof(float) * 2 * c;
  const int staged = smem <= 32 * 1024 && (norm.mean || e.scale || e.shift) ? 1 : 0;
  if (norm.mean && !staged) return PCE_ERR_UNSUPPORTED;
  // enough blocks for every thread to have one round of pieces, as many as are resident
  const long long want = (total / kVec + 4 * 256 - 1) / (4 * 256);
  const int sms = device_sm_count();
  int grid = static_cast<int>(std::max<long long>(1, std::min<long long>(want, static_cast<long long>(sms) * (e.residual ? 3 : 4))));
  const int row_pieces = c / kVec;
  int unit = row_pieces;  // blocks whose pieces make whole rows: row_pieces / gcd(row_pieces, 256)
  while (unit > 0 && unit % 2 == 0 && row_pieces / unit < 256) unit /= 2;
  const int mode = c % kVec ? 2 : (staged && grid >= unit ? 0 : 1);
  if (mode == 0) grid = grid / unit * unit;
  const size_t bytes = staged ? smem : 0;
#define PCE_AFFINE(M)                                                                                       \
  do {                                                                                                      \
    if (e.residual)                                                                                         \
      k_scale_shift_act<T, M, true><<<grid, 256, bytes, st>>>(x_t, total, c, y_t, e, norm, staged);         \
    else                                                                                                    \
      k_scale_shift_act<T, M, false><<<grid, 256, bytes, st>>>(x_t, total, c, y_t, e, norm, staged);        \
  } while (0)
  if (mode == 0) PCE_AFFINE(0); else if (mode == 1) PCE_AFFINE(1); else PCE_AFFINE(2);
#undef PCE_AFFINE
  PCE_LAUNCH_CHECK();
  return PCE_OK;
}

template <typename T>
static int launch_simt(const void* in, const void* w, const uint32_t* mask, const int* rowptr, const int* nbr,
                       int n_out, int cin, int cout, int kv, void* out, const EpiDev& ep, bool ident,
                       cudaStream_t st) {
  if (n_out == 0) return PCE_OK;
  int need = (cout + 3) / 4;
  int g = 1;
  while (g < need && g < 32) g <<= 1;
  const int vec_in = sizeof(T) == 4 ? 4 : 8;
  // 16-byte pieces of the input rows, four weights at a time: of widths that allow it, from addresses that do
  const bool vec = (cin % vec_in == 0) && (cout % 4 == 0) && reinterpret_cast<uintptr_t>(in) % 16 == 0 &&
                   reinterpret_cast<uintptr_t>(w) % (4 * sizeof(T)) == 0;
  const int rows_per_block = 256 / g;
  const int grid = div_up(n_out, rows_per_block);
  const T* in_t = static_cast<const T*>(in);
  const T* w_t = static_cast<const T*>(w);
  T* out_t = static_cast<T*>(out);
#define PCE_SIMT_LAUNCH(V, I) \
  k_conv_simt<T, V, I><<<grid, 256, 0, st>>>(in_t, w_t, mask, rowptr, nbr, n_out, cin, cout, kv, out_t, ep, g)
  if (vec) {
    if (ident)
      PCE_SIMT_LAUNCH(true, true);
    else
      PCE_SIMT_LAUNCH(true, false);
  } else {
    if (ident)
      PCE_SIMT_LAUNCH(false, true);
    else
      PCE_SIMT_LAUNCH(false, false);
  }
#undef PCE_SIMT_LAUNCH
  PCE_LAUNCH_CHECK();
  return PCE_OK;
}

int conv_simt(const void* in, const void* w, const uint32_t* mask, const int* rowptr, const int* nbr, int n_out,
              int cin, int cout, int kv, void* out, int dtype, const pce_epilogue* ep, bool ident,
              cudaStream_t st) {
  EpiDev e = to_dev(ep);
  if (dtype == PCE_F32)
    return launch_simt<float>(in, w, mask, rowptr, nbr, n_out, cin, cout, kv, out, e, ident, st);
  if (dtype == PCE_F16)
    return launch_simt<__half>(in, w, mask, rowptr, nbr, n_out, cin, cout, kv, out, e, ident, st);
  return PCE_ERR_UNSUPPORTED;
}

// Rows rows[i] (or i where rows == nullptr) of a row-major matrix, copied into consecutive rows of `dst` in
// 16-byte pieces.  `dst` may be another GPU's memory mapped into this process: plain stores, no loads from it.
__global__ void k_push_rows(const char* __restrict__ src, long long src_pitch, const int* __restrict__ rows, int n_rows,
                            int pieces, char* __restrict__ dst, long long dst_pitch) {
  const long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
  if (i >= static_cast<long long>(n_rows) * pieces) return;
  const int r = static_cast<int>(i / pieces), p = static_cast<int>(i % pieces);
  const long long from = rows ? __ldg(rows + r) : r;
  const uint4 v = *reinterpret_cast<const uint4*>(src + from * src_pitch + 16ll * p);
  *reinterpret_cast<uint4*>(dst + r * dst_pitch + 16ll * p) = v;
}

}  // namespace pce

using namespace pce;

extern "C" {

int pce_push_rows(const void* src, int64_t src_pitch_bytes, const int32_t* rows, int32_t n_rows, int32_t row_bytes,
                  void* dst, int64_t dst_pitch_bytes, void* stream) {
  if (n_rows < 0 || row_bytes < 16 || (row_bytes & 15) || src_pitch_bytes < row_bytes || dst_pitch_bytes < row_bytes ||
      (src_pitch_bytes & 15) || (dst_pitch_bytes & 15))
    return PCE_ERR_INVALID;
  if (n_rows == 0) return PCE_OK;
  if (!src || !dst || ((reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst)) & 15)) return PCE_ERR_INVALID;
  const int pieces = row_bytes / 16;
  const long long total = static_cast<long long>(n_rows) * pieces;
  k_push_rows<<<static_cast<unsigned>((total + 255) / 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const char*>(src), src_pitch_bytes, rows, n_rows, pieces, static_cast<char*>(dst), dst_pitch_bytes);
  PCE_LAUNCH_CHECK();
  return PCE_OK;
}

int pce_scale_shift_act(const void* x, int64_t n, int32_t c, void* y, int32_t dtype, const pce_epilogue* ep,
                        void* stream) {
  if (n < 0 || c < 1) return PCE_ERR_INVALID;
  if (n == 0) return PCE_OK;
  if (!x || !y) return PCE_ERR_INVALID;
  if (ep && (ep->extra_feats || ep->push_slot[0] || ep->push_slot[1] || (ep->in_ld > 0 && ep->in_ld != c) ||
             (ep->out_ld > 0 && ep->out_ld != c)))
    return PCE_ERR_UNSUPPORTED;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  EpiDev e = to_dev(ep);
  const long long total = static_cast<long long>(n) * c;
  const NormSrc none{nullptr, nullptr, nullptr, nullptr, 0.f, 0};
  if (dtype == PCE_F32) return launch_affine<float>(x, total, c, y, e, none, st);
  if (dtype == PCE_F16) return launch_affine<__half>(x, total, c, y, e, none, st);
  return PCE_ERR_UNSUPPORTED;
}

int pce_batchnorm(const void* x, int64_t n, int32_t c, void* y, int32_t dtype, const void* mean, const void* var,
                  const void* gamma, const void* beta, int32_t param_dtype, float eps, void* stream) {
  if (n < 0 || c < 1 || !mean || !var) return PCE_ERR_INVALID;
  if (param_dtype != PCE_F32 && param_dtype != PCE_F16) return PCE_ERR_UNSUPPORTED;
  if (n == 0) return PCE_OK;
  if (!x || !y) return PCE_ERR_INVALID;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const EpiDev e{nullptr, nullptr, nullptr, PCE_ACT_NONE, 0.f};
  const NormSrc norm{mean, var, gamma, beta, eps, param_dtype == PCE_F16 ? 1 : 0};
  const long long total = static_cast<long long>(n) * c;
  if (dtype == PCE_F32) return launch_affine<float>(x, total, c, y, e, norm, st);
  if (dtype == PCE_F16) return launch_affine<__half>(x, total, c, y, e, norm, st);
  return PCE_ERR_UNSUPPORTED;
}

}  // extern "C"

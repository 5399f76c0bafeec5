// LayerNorm forward/backward, GELU forward/backward, and microbatch BatchNorm (channels-last) kernels, sm_100a.
//
// Reference call sites: ViT / BERT blocks (`benchmarks/moco-v3/vits.py:132`, `benchmarks/distilbert/bert.py`),
// GELU inside their MLPs, and the microbatch-aware BatchNorm (`tspipe/batchnorm.py:45-120`), all plain ATen calls
// there.  Under bf16 autocast ATen's layer_norm up-casts to fp32 and writes fp32; these kernels read and write
// the activation dtype directly and keep statistics in fp32.
#include "common.cuh"
#include "gelu.cuh"
#include "tspipe_kernels.h"

namespace {

constexpr int kLnMaxVec = 4;   // per-lane register tile: 4 x 8 elements -> rows up to 1024 wide stay in registers

// ---------------------------------------------------------------------------------------------
// LayerNorm forward: one warp per row, NV 16-byte vectors per lane (rows of up to 256 * NV elements), single pass from
// registers.  Each warp loads two rows before it reduces the first.  ADD: the rows are x + a, rounded to T and written to
// `sum` as the separate addition would (residual connections: one read and one launch less).
// ---------------------------------------------------------------------------------------------
template <typename T, int NV, bool ADD>
__global__ void __launch_bounds__(128) ln_fwd_kernel(const T* __restrict__ x, const T* __restrict__ a, T* __restrict__ sum,
                                                     const float* __restrict__ w,
                                                     const float* __restrict__ b, T* __restrict__ y,
                                                     float* __restrict__ mean, float* __restrict__ rstd, int rows,
                                                     int d, float eps) {
  tsp::let_next_start();
  constexpr int R = 2;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int row0 = (blockIdx.x * 4 + warp) * R;
  const int nvec = d >> 3;
  tsp::Raw8<T> raw[R][NV], add[ADD ? R : 1][ADD ? NV : 1];
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int k = 0; k < NV; ++k)
      if (row0 + r < rows && lane + 32 * k < nvec) {
        const int64_t at = (int64_t)(row0 + r) * d + (lane + 32 * k) * 8;
        tsp::ldraw(x, at, raw[r][k]);
        if constexpr (ADD) tsp::ldraw(a, at, add[r][k]);
      }
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int row = row0 + r;
    if (row >= rows) return;
    float v[NV][8];
    float s = 0.f;
#pragma unroll
    for (int k = 0; k < NV; ++k)
      if (lane + 32 * k < nvec) {
        tsp::cvt8(raw[r][k], v[k]);
        if constexpr (ADD) {
          float av[8];
          tsp::cvt8(add[r][k], av);
#pragma unroll
          for (int e = 0; e < 8; ++e) v[k][e] += av[e];
          tsp::round_as<T>(v[k]);
          if (sum != nullptr) tsp::st8(sum, (int64_t)row * d + (lane + 32 * k) * 8, v[k]);
        }
#pragma unroll
        for (int e = 0; e < 8; ++e) s += v[k][e];
      }
    const float mu = tsp::warp_sum(s) / d;
    float q = 0.f;
#pragma unroll
    for (int k = 0; k < NV; ++k)
      if (lane + 32 * k < nvec) {
#pragma unroll
        for (int e = 0; e < 8; ++e) { const float c = v[k][e] - mu; q += c * c; }
      }
    const float rs = rsqrtf(tsp::warp_sum(q) / d + eps);
    if (lane == 0) { mean[row] = mu; rstd[row] = rs; }
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      const int vi = lane + 32 * k;
      if (vi < nvec) {
        float wv[8], bv[8], o[8];
        tsp::ld8(w, (int64_t)vi * 8, wv);
        tsp::ld8(b, (int64_t)vi * 8, bv);
#pragma unroll
        for (int e = 0; e < 8; ++e) o[e] = (v[k][e] - mu) * rs * wv[e] + bv[e];
        tsp::st8(y + (int64_t)row * d, (int64_t)vi * 8, o);
      }
    }
  }
}

// LayerNorm backward: dx per row (one warp per row) and the block's partial dw / db from ONE read of dy and x, bound by
// memory.  A lane keeps its columns' dw / db sums in registers over all rows of its warp and holds the row as loaded (16
// bits where the activation has 16 bits), so that 16 warps fit an SM; an earlier one-kernel form with the row in fp32 took
// 176 registers and ran at 1.45 TB/s, and separate dx and dw / db kernels read everything twice.  [12608, 768] bf16,
// B200, with its reduction (3): 40 us as separate kernels, 23 this way, with a residual's gradient 26, and 33 where that was loaded
// behind the sums.  (Requesting the next row ahead of the current one: 36, fewer warps fit.)
// partial layout: [gridDim.x][2][d] fp32 (scratch memory owned by the caller), summed by ln_bwd_reduce_kernel.
constexpr int kLnBwdWarps = 8;
// ADD: `skip` (the gradient that reaches the row on a residual connection) is added to the rounded dx.
template <typename T, int NV, bool ADD>
__global__ void __launch_bounds__(kLnBwdWarps * 32, sizeof(T) == 2 ? 2 : 1)
ln_bwd_kernel(const T* __restrict__ dy, const T* __restrict__ x, const T* __restrict__ skip, const float* __restrict__ w,
              const float* __restrict__ mean, const float* __restrict__ rstd, T* __restrict__ dx,
              float* __restrict__ partial, int rows, int d) {
  tsp::let_next_start();
  __shared__ float sm[2 * 256 * NV];       // [2][256 * NV] the block's sums
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nvec = d >> 3;
  float adw[NV][8], adb[NV][8];
#pragma unroll
  for (int k = 0; k < NV; ++k)
#pragma unroll
    for (int e = 0; e < 8; ++e) { adw[k][e] = 0.f; adb[k][e] = 0.f; }
  for (int row = blockIdx.x * kLnBwdWarps + warp; row < rows; row += gridDim.x * kLnBwdWarps) {
    tsp::Raw8<T> xr[NV], gr[NV], kr[ADD ? NV : 1];
#pragma unroll
    for (int k = 0; k < NV; ++k)
      if (lane + 32 * k < nvec) {
        const int64_t at = (int64_t)row * d + (lane + 32 * k) * 8;
        tsp::ldraw(x, at, xr[k]);
        tsp::ldraw(dy, at, gr[k]);
        if constexpr (ADD) tsp::ldraw(skip, at, kr[k]);
      }
    const float mu = mean[row], rs = rstd[row];
    float s1 = 0.f, s2 = 0.f;
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      const int vi = lane + 32 * k;
      if (vi < nvec) {
        float xv[8], gv[8], wv[8];
        tsp::cvt8(xr[k], xv);
        tsp::cvt8(gr[k], gv);
        tsp::ld8(w, (int64_t)vi * 8, wv);
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const float xh = (xv[e] - mu) * rs, gw = gv[e] * wv[e];
          s1 += gw;
          s2 += gw * xh;
          adw[k][e] += gv[e] * xh;
          adb[k][e] += gv[e];
        }
      }
    }
    s1 = tsp::warp_sum(s1) / d;
    s2 = tsp::warp_sum(s2) / d;
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      const int vi = lane + 32 * k;
      if (vi < nvec) {
        float xv[8], gv[8], wv[8], o[8];
        tsp::cvt8(xr[k], xv);
        tsp::cvt8(gr[k], gv);
        tsp::ld8(w, (int64_t)vi * 8, wv);
#pragma unroll
        for (int e = 0; e < 8; ++e) o[e] = rs * (gv[e] * wv[e] - s1 - (xv[e] - mu) * rs * s2);
        if constexpr (ADD) {
          float sv[8];
          tsp::cvt8(kr[k], sv);
          tsp::round_as<T>(o);
#pragma unroll
          for (int e = 0; e < 8; ++e) o[e] += sv[e];
        }
        tsp::st8(dx + (int64_t)row * d, (int64_t)vi * 8, o);
      }
    }
  }
  // the warps add their sums in turn: no atomics, one order.  Value e of vector vi sits at [e][vi] (conflict-free).
  for (int turn = 0; turn < kLnBwdWarps; ++turn) {
    if (warp == turn) {
#pragma unroll
      for (int k = 0; k < NV; ++k)
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          float* p = sm + e * 32 * NV + 32 * k + lane;
          p[0] = (turn ? p[0] : 0.f) + adw[k][e];
          p[256 * NV] = (turn ? p[256 * NV] : 0.f) + adb[k][e];
        }
    }
    __syncthreads();
  }
  float* out = partial + (int64_t)blockIdx.x * 2 * d;
  for (int i = threadIdx.x; i < d; i += blockDim.x) {
    const float* p = sm + (i & 7) * 32 * NV + (i >> 3);
    out[i] = p[0];
    out[d + i] = p[256 * NV];
  }
}

// part 2: dw[j] = sum_blocks partial[b][0][j], db likewise.  Block = 32 columns x kLnReduce slices of the blocks.
constexpr int kLnReduce = 32;
__global__ void __launch_bounds__(32 * kLnReduce) ln_bwd_reduce_kernel(const float* __restrict__ partial, int nblocks, int d,
                                                            float* __restrict__ dw, float* __restrict__ db, int add) {
  tsp::let_next_start();
  __shared__ float sm[kLnReduce][33];
  const int lane = threadIdx.x & 31, slice = threadIdx.x >> 5;
  const int j = blockIdx.x * 32 + lane;
  float acc = 0.f;
  if (j < 2 * d) {
#pragma unroll 4
    for (int b = slice; b < nblocks; b += kLnReduce) acc += partial[(int64_t)b * 2 * d + j];
  }
  sm[slice][lane] = acc;
  __syncthreads();
  const float total = tsp::warp_sum(sm[lane][slice]);       // warp = column, lane = slice
  __syncthreads();
  if (lane == 0) sm[0][slice] = total;
  __syncthreads();
  if (slice == 0 && j < 2 * d) {
    acc = sm[0][lane];
    float* out = j < d ? dw + j : db + (j - d);
    *out = add ? *out + acc : acc;
  }
}

// ---------------------------------------------------------------------------------------------
// GELU (erf form), optionally with the bias add in front: y = gelu(x + bias)
// ---------------------------------------------------------------------------------------------
// Bound by memory once the arithmetic is about 20 instructions per element.  The grid stride is a multiple of a row
// (gelu_blocks), so a thread keeps the eight bias values of its columns in registers; U vectors in flight per thread.
// [12608, 3072] bf16, B200, forward 59 us and backward 62 with the
// correctly rounded reciprocal and exponential and an index remainder per vector, 33 and 41 this way.
constexpr int kGeluFwdVecs = 4, kGeluBwdVecs = 2;

template <typename T>
__global__ void __launch_bounds__(256) gelu_fwd_kernel(const T* __restrict__ x, const float* __restrict__ bias,
                                                       T* __restrict__ y, int64_t n, int d) {
  tsp::let_next_start();
  constexpr int U = kGeluFwdVecs;
  const int64_t nv = n >> 3;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  const uint32_t first = blockIdx.x * blockDim.x + threadIdx.x;
  float b[8] = {};
  if (bias) tsp::ld8(bias, (int64_t)(first % (uint32_t)(d >> 3)) * 8, b);
  for (int64_t i = first; i < nv; i += U * stride) {
    tsp::Raw8<T> raw[U];
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (i + u * stride < nv) tsp::ldraw(x, (i + u * stride) * 8, raw[u]);
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (i + u * stride < nv) {
        float v[8];
        tsp::cvt8(raw[u], v);
        tsp::gelu_all<T>(v, b);
        tsp::st8(y, (i + u * stride) * 8, v);
      }
  }
}

template <typename T>
__global__ void __launch_bounds__(256) gelu_bwd_kernel(const T* __restrict__ dy, const T* __restrict__ x,
                                                       const float* __restrict__ bias, T* __restrict__ dx, int64_t n,
                                                       int d) {
  tsp::let_next_start();
  constexpr int U = kGeluBwdVecs;
  const int64_t nv = n >> 3;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  const uint32_t first = blockIdx.x * blockDim.x + threadIdx.x;
  float b[8] = {};
  if (bias) tsp::ld8(bias, (int64_t)(first % (uint32_t)(d >> 3)) * 8, b);
  for (int64_t i = first; i < nv; i += U * stride) {
    tsp::Raw8<T> xr[U], gr[U];
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (i + u * stride < nv) { tsp::ldraw(x, (i + u * stride) * 8, xr[u]); tsp::ldraw(dy, (i + u * stride) * 8, gr[u]); }
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (i + u * stride < nv) {
        float v[8], g[8];
        tsp::cvt8(xr[u], v);
        tsp::cvt8(gr[u], g);
        tsp::times_gelu_grad<T>(g, v, b);
        tsp::st8(dx, (i + u * stride) * 8, g);
      }
  }
}

// The same with the column sums of dx (the gradient of the bias), of the values as they are stored: 32 lanes = 256 columns of a
// row, eight warps = eight rows, blocks stacked over the rows, so that a thread keeps its columns' sums in registers and a
// block adds one number per column.  [12608, 3072] bf16: 41 us and a pass of 16 for the sums, 48 this way.  x and dy are read with
// evict-first hints, so that dx is in the L2 cache for the two products that follow; with a reader of dx behind it 75.8 us without
// hints and 67.6 with, [12608, 4096] 108.6 and 94.2, [4000, 3072] 40.1 and 38.7, [50432, 3072] 250 both.
constexpr int kGeluSumRows = 8, kGeluSumVecs = 2;

template <typename T>
__global__ void __launch_bounds__(256) gelu_bwd_sums_kernel(const T* __restrict__ dy, const T* __restrict__ x,
                                                            const float* __restrict__ bias, T* __restrict__ dx,
                                                            float* __restrict__ sums, int64_t rows, int d) {
  tsp::let_next_start();
  constexpr int U = kGeluSumVecs;
  __shared__ float part[kGeluSumRows][256 + 8];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int col = (blockIdx.x * 32 + lane) * 8;
  const bool in = col < d;
  float b[8] = {}, acc[8] = {};
  if (in) tsp::ld8(bias, (int64_t)col, b);
  const int64_t step = (int64_t)gridDim.y * kGeluSumRows;
  for (int64_t r = (int64_t)blockIdx.y * kGeluSumRows + warp; in && r < rows; r += U * step) {
    tsp::Raw8<T> xr[U], gr[U];
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (r + u * step < rows) { tsp::ldraw<true>(x, (r + u * step) * d + col, xr[u]); tsp::ldraw<true>(dy, (r + u * step) * d + col, gr[u]); }
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (r + u * step < rows) {
        float v[8], g[8];
        tsp::cvt8(xr[u], v);
        tsp::cvt8(gr[u], g);
        tsp::times_gelu_grad<T>(g, v, b);
        tsp::round_as<T>(g);
        tsp::st8(dx, (r + u * step) * d + col, g);
#pragma unroll
        for (int e = 0; e < 8; ++e) acc[e] += g[e];
      }
  }
#pragma unroll
  for (int e = 0; e < 8; ++e) part[warp][lane * 8 + e] = acc[e];
  __syncthreads();
  const int c = blockIdx.x * 256 + threadIdx.x;
  if (c < d) {
    float v = 0.f;
#pragma unroll
    for (int k = 0; k < kGeluSumRows; ++k) v += part[k][threadIdx.x];
    atomicAdd(sums + c, v);
  }
}

template <typename T, bool ADD>
int launch_ln_fwd(const void* x, const void* a, void* sum, const float* w, const float* b, void* y, float* mean, float* rstd,
                  int rows, int d, float eps, cudaStream_t stream) {
  const int grid = (rows + 7) / 8;
#define TSP_LN(NV)                                                                                                       \
  ln_fwd_kernel<T, NV, ADD><<<grid, 128, 0, stream>>>((const T*)x, (const T*)a, (T*)sum, w, b, (T*)y, mean, rstd, rows, d, \
                                                      eps)
  if (d <= 256) TSP_LN(1);
  else if (d <= 512) TSP_LN(2);
  else if (d <= 768) TSP_LN(3);
  else TSP_LN(4);
#undef TSP_LN
  return TSP_LAUNCH_CHECK();
}

template <typename T, bool ADD>
int launch_ln_bwd(const void* dy, const void* x, const void* skip, const float* w, const float* mean, const float* rstd,
                  void* dx, float* dw, float* db, float* partial, int rows, int d, int nb, int add, cudaStream_t stream) {
#define TSP_LN(NV)                                                                                                    \
  ln_bwd_kernel<T, NV, ADD><<<nb, kLnBwdWarps * 32, 0, stream>>>((const T*)dy, (const T*)x, (const T*)skip, w, mean, rstd, \
                                                                 (T*)dx, partial, rows, d)
  if (d <= 256) TSP_LN(1);
  else if (d <= 512) TSP_LN(2);
  else if (d <= 768) TSP_LN(3);
  else TSP_LN(4);
#undef TSP_LN
  ln_bwd_reduce_kernel<<<(2 * d + 31) / 32, 32 * kLnReduce, 0, stream>>>(partial, nb, d, dw, db, add);
  return TSP_LAUNCH_CHECK();
}

}  // namespace

extern "C" {

int tsp_layernorm_fwd(const void* x, const float* w, const float* b, void* y, float* mean, float* rstd, int rows, int d,
                      float eps, int dtype, cudaStream_t stream) {
  if (rows <= 0) return 0;
  if (d % 8 != 0 || d > 8 * 32 * kLnMaxVec) return -3;
  if ((((uintptr_t)w | (uintptr_t)b) & 15) != 0) return -2;            // (read 16 bytes at a time)
  return dtype == TSP_DTYPE_BF16
             ? launch_ln_fwd<__nv_bfloat16, false>(x, nullptr, nullptr, w, b, y, mean, rstd, rows, d, eps, stream)
             : launch_ln_fwd<float, false>(x, nullptr, nullptr, w, b, y, mean, rstd, rows, d, eps, stream);
}

// sum = x + a (rounded; optional), y = LayerNorm(sum).
int tsp_add_layernorm_fwd(const void* x, const void* a, void* sum, const float* w, const float* b, void* y, float* mean,
                          float* rstd, int rows, int d, float eps, int dtype, cudaStream_t stream) {
  if (rows <= 0) return 0;
  if (d % 8 != 0 || d > 8 * 32 * kLnMaxVec) return -3;
  if ((((uintptr_t)w | (uintptr_t)b) & 15) != 0) return -2;            // (read 16 bytes at a time)
  return dtype == TSP_DTYPE_BF16 ? launch_ln_fwd<__nv_bfloat16, true>(x, a, sum, w, b, y, mean, rstd, rows, d, eps, stream)
                                 : launch_ln_fwd<float, true>(x, a, sum, w, b, y, mean, rstd, rows, d, eps, stream);
}

// Two blocks per SM, at least two rows per warp.
int tsp_layernorm_bwd_blocks(int rows) {
  const int nb = (rows + 2 * kLnBwdWarps - 1) / (2 * kLnBwdWarps);
  const int cap = 148 * 2;
  return nb > cap ? cap : (nb < 1 ? 1 : nb);
}

// `partial` is scratch of tsp_layernorm_bwd_blocks(rows) * 2 * d floats; `skip` (optional, dx's shape) is added to dx;
// `add`: dw and db are added to instead of set.
int tsp_layernorm_bwd_add(const void* dy, const void* x, const void* skip, const float* w, const float* mean, const float* rstd, void* dx,
                          float* dw, float* db, float* partial, int rows, int d, int dtype, int add,
                          cudaStream_t stream) {
  if (rows <= 0) return 0;
  if (d % 8 != 0 || d > 8 * 32 * kLnMaxVec) return -3;
  if (((uintptr_t)w & 15) != 0) return -2;
  const int nb = tsp_layernorm_bwd_blocks(rows);
#define TSP_LN(T, ADD) launch_ln_bwd<T, ADD>(dy, x, skip, w, mean, rstd, dx, dw, db, partial, rows, d, nb, add, stream)
  if (dtype == TSP_DTYPE_BF16) return skip != nullptr ? TSP_LN(__nv_bfloat16, true) : TSP_LN(__nv_bfloat16, false);
  return skip != nullptr ? TSP_LN(float, true) : TSP_LN(float, false);
#undef TSP_LN
}

int tsp_layernorm_bwd(const void* dy, const void* x, const float* w, const float* mean, const float* rstd, void* dx,
                      float* dw, float* db, float* partial, int rows, int d, int dtype, cudaStream_t stream) {
  return tsp_layernorm_bwd_add(dy, x, nullptr, w, mean, rstd, dx, dw, db, partial, rows, d, dtype, 0, stream);
}

// Blocks of the GELU passes: `per_thread` vectors per thread on large tensors, at most eight blocks per SM, rounded so
// that the grid stride is a multiple of a row of the bias.
static int gelu_blocks(int64_t nv, int cpv, int per_thread) {
  return tsp::row_stride_blocks(nv, cpv, 256, per_thread, 148 * 2, 148 * 8);
}

int tsp_gelu_fwd(const void* x, const float* bias, void* y, int64_t n, int d, int dtype, cudaStream_t stream) {
  if (n <= 0) return 0;
  if (n % 8 != 0 || (bias && d % 8 != 0)) return -3;
  if (((uintptr_t)bias & 15) != 0) return -2;
  const int blocks = gelu_blocks(n / 8, bias ? d / 8 : 1, kGeluFwdVecs);
  if (dtype == TSP_DTYPE_BF16)
    gelu_fwd_kernel<__nv_bfloat16><<<blocks, 256, 0, stream>>>((const __nv_bfloat16*)x, bias, (__nv_bfloat16*)y, n, d);
  else
    gelu_fwd_kernel<float><<<blocks, 256, 0, stream>>>((const float*)x, bias, (float*)y, n, d);
  return TSP_LAUNCH_CHECK();
}

int tsp_gelu_bwd(const void* dy, const void* x, const float* bias, void* dx, int64_t n, int d, int dtype,
                 cudaStream_t stream) {
  if (n <= 0) return 0;
  if (n % 8 != 0 || (bias && d % 8 != 0)) return -3;
  if (((uintptr_t)bias & 15) != 0) return -2;
  const int blocks = gelu_blocks(n / 8, bias ? d / 8 : 1, kGeluBwdVecs);
  if (dtype == TSP_DTYPE_BF16)
    gelu_bwd_kernel<__nv_bfloat16><<<blocks, 256, 0, stream>>>((const __nv_bfloat16*)dy, (const __nv_bfloat16*)x, bias,
                                                               (__nv_bfloat16*)dx, n, d);
  else
    gelu_bwd_kernel<float><<<blocks, 256, 0, stream>>>((const float*)dy, (const float*)x, bias, (float*)dx, n, d);
  return TSP_LAUNCH_CHECK();
}

// Also adds the column sums of dx [rows, d] to sums [d] (fp32).  d % 8 == 0, bias 16-byte aligned.
int tsp_gelu_bwd_sums(const void* dy, const void* x, const float* bias, void* dx, float* sums, int64_t rows, int d, int dtype,
                      cudaStream_t stream) {
  if (rows <= 0 || d <= 0) return 0;
  if (d % 8 != 0) return -3;
  if (bias == nullptr || ((uintptr_t)bias & 15) != 0) return -2;
  const int slabs = (d + 255) / 256;
  int64_t blocks = (rows + kGeluSumRows * kGeluSumVecs - 1) / (kGeluSumRows * kGeluSumVecs);
  int sms = 0;
  if (cudaError_t e = tsp::usable_sms(sms); e != cudaSuccess) return (int)e;
  const int64_t most = (sms * 6 + slabs - 1) / slabs;                  // six blocks per SM
  if (blocks > most) blocks = most;
  const dim3 grid((unsigned)slabs, (unsigned)blocks);
  if (dtype == TSP_DTYPE_BF16)
    gelu_bwd_sums_kernel<__nv_bfloat16><<<grid, 256, 0, stream>>>((const __nv_bfloat16*)dy, (const __nv_bfloat16*)x, bias,
                                                                  (__nv_bfloat16*)dx, sums, rows, d);
  else
    gelu_bwd_sums_kernel<float><<<grid, 256, 0, stream>>>((const float*)dy, (const float*)x, bias, (float*)dx, sums, rows, d);
  return TSP_LAUNCH_CHECK();
}

// ---------------------------------------------------------------------------------------------
// LayerNorm backward for callers that must not allocate (see tspipe_noalloc.h).
// The per-block dw/db partial sums go to this fixed array instead of a caller-provided buffer.
// Every GPU that loads the library holds these 1.16 MiB until the process exits.
// ---------------------------------------------------------------------------------------------
#include "tspipe_noalloc.h"

static __device__ __align__(256) float g_ln_bwd_scratch[TSP_NOALLOC_LN_MAX_BLOCKS * 2 * TSP_NOALLOC_LN_MAX_D];

int tsp_layernorm_bwd_noalloc(const void* dy, const void* x, const float* w, const float* mean, const float* rstd,
                              void* dx, float* dw, float* db, int rows, int d, int dtype, cudaStream_t stream) {
  // In host code `g_ln_bwd_scratch` is only a handle for the runtime, not an address a kernel can use: the
  // device address has to be looked up, once per device, with that device current.
  static float* scratch_of_device[TSP_NOALLOC_MAX_DEVICES] = {nullptr};
  if (rows < 0 || d <= 0) return -3;
  if (rows == 0) return 0;
  if (d % 8 != 0) return -3;
  if (d > TSP_NOALLOC_LN_MAX_D) return TSP_NOALLOC_ERR_TOO_LARGE;
  if (dtype != TSP_DTYPE_F32 && dtype != TSP_DTYPE_BF16) return -3;
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return (int)e;
  if (dev < 0 || dev >= TSP_NOALLOC_MAX_DEVICES) return TSP_NOALLOC_ERR_TOO_LARGE;
  float* scratch = scratch_of_device[dev];
  if (scratch == nullptr) {
    e = cudaGetSymbolAddress((void**)&scratch, g_ln_bwd_scratch);
    if (e != cudaSuccess) return (int)e;
    scratch_of_device[dev] = scratch;
  }
  int nb = tsp_layernorm_bwd_blocks(rows);
  if (nb > TSP_NOALLOC_LN_MAX_BLOCKS) nb = TSP_NOALLOC_LN_MAX_BLOCKS;
  // Nothing in the scratch has to start at zero: each of the nb blocks overwrites its whole 2*d slice and the
  // reduction reads exactly those nb slices, so what an earlier call left behind is never read.
  return dtype == TSP_DTYPE_BF16
             ? launch_ln_bwd<__nv_bfloat16, false>(dy, x, nullptr, w, mean, rstd, dx, dw, db, scratch, rows, d, nb, 0, stream)
             : launch_ln_bwd<float, false>(dy, x, nullptr, w, mean, rstd, dx, dw, db, scratch, rows, d, nb, 0, stream);
}

}  // extern "C"

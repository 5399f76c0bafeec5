// Fused loss kernels (forward value + gradient in one launch), sm_100a.
//
// Reference math: BYOL regression `benchmarks/byol/trainer.py:51-55,192-196`; soft-target KD
// `benchmarks/soft_target/kd_losses/st.py:18-23` + CE `benchmarks/soft_target/train_kd.py:448-453`;
// DistilBERT KL/MLM-CE terms `benchmarks/distilbert/distiller.py:711-772`.  The reference evaluates each with
// 5-10 library ops (normalize, softmax, log_softmax, kl_div, cross_entropy, masked_select copies) and a
// second sweep in autograd; the loss GPU holds the whole mini-batch, so these are latency- and
// bandwidth-bound row kernels: one read of the rows (teacher rows may sit behind a peer pointer), one write of
// the student gradient.
#include "common.cuh"
#include "tspipe_kernels.h"

namespace {

// V consecutive elements of a row (V = 8: one 16-byte access per 8 bf16; V = 1: any alignment).  Gradients are written
// once and read by another launch: streaming stores keep the rows that the second sweep reads again in L2.
template <typename T, int V>
__device__ __forceinline__ void load_part(const T* __restrict__ row, int i, float (&v)[V]) {
  if constexpr (V == 8) tsp::ld8(row, (int64_t)i * 8, v);
  else v[0] = tsp::ld(row, i);
}
__device__ __forceinline__ void stream8(float* p, const float (&v)[8]) {
  __stcs(reinterpret_cast<float4*>(p), make_float4(v[0], v[1], v[2], v[3]));
  __stcs(reinterpret_cast<float4*>(p) + 1, make_float4(v[4], v[5], v[6], v[7]));
}
__device__ __forceinline__ void stream8(__nv_bfloat16* p, const float (&v)[8]) {
  uint4 raw;
  __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&raw);
#pragma unroll
  for (int k = 0; k < 4; ++k) h[k] = __floats2bfloat162_rn(v[2 * k], v[2 * k + 1]);
  __stcs(reinterpret_cast<uint4*>(p), raw);
}
template <typename T, int V>
__device__ __forceinline__ void store_part(T* __restrict__ row, int i, const float (&v)[V]) {
  if constexpr (V == 8) stream8(row + (int64_t)i * 8, v);
  else tsp::st(row, i, v[0]);
}

// ---------------------------------------------------------------------------------------------
// BYOL: loss += scale * sum_rows (2 - 2 cos(x_r, y_r)) ; gx = scale * d/dx
// one warp per row, 8 elements per lane and access when the rows allow it (VEC).  blockIdx.y = pair: both directions
// of the symmetric loss go out as one launch; pair p reads x[p], y[p] and writes gx + p * n * d.  A few microseconds of
// work, so launches are what it costs: forward and backward of both directions of [128, 256] took 186 us with a launch and
// four library kernels per direction and take 113.
// ---------------------------------------------------------------------------------------------
template <typename T>
struct PairPtrs {
  const T* x[2];
  const T* y[2];
};
template <typename T, bool VEC>
__global__ void __launch_bounds__(128) byol_kernel(const PairPtrs<T> in, int n, int d, float scale, double* __restrict__ sum,
                                                   float* __restrict__ loss, T* __restrict__ gx) {
  constexpr int V = VEC ? 8 : 1;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int row = blockIdx.x * 4 + warp;
  float contrib = 0.f;
  if (row < n) {
    const T* xr = (blockIdx.y ? in.x[1] : in.x[0]) + (int64_t)row * d;
    const T* yr = (blockIdx.y ? in.y[1] : in.y[0]) + (int64_t)row * d;
    float xx = 0.f, yy = 0.f, xy = 0.f;
    const int nv = d / V;
    for (int i = lane; i < nv; i += 32) {
      float a[V], b[V];
      load_part<T, V>(xr, i, a);
      load_part<T, V>(yr, i, b);
#pragma unroll
      for (int e = 0; e < V; ++e) { xx += a[e] * a[e]; yy += b[e] * b[e]; xy += a[e] * b[e]; }
    }
    xx = tsp::warp_sum(xx); yy = tsp::warp_sum(yy); xy = tsp::warp_sum(xy);
    const float nx = fmaxf(sqrtf(xx), 1e-12f), ny = fmaxf(sqrtf(yy), 1e-12f);
    const float cosv = xy / (nx * ny);
    contrib = 2.f - 2.f * cosv;
    if (gx != nullptr) {
      T* gr = gx + ((int64_t)blockIdx.y * n + row) * d;
      const float c1 = -2.f * scale / (nx * ny), c2 = 2.f * scale * cosv / (nx * nx);
      for (int i = lane; i < nv; i += 32) {
        float a[V], b[V];
        load_part<T, V>(xr, i, a);
        load_part<T, V>(yr, i, b);
#pragma unroll
        for (int e = 0; e < V; ++e) a[e] = c1 * b[e] + c2 * a[e];
        store_part<T, V>(gr, i, a);
      }
    }
  }
  __shared__ float part[4];
  if (lane == 0) part[warp] = contrib;
  __syncthreads();
  if (threadIdx.x == 0) {
    const float v = part[0] + part[1] + part[2] + part[3];
    if (sum == nullptr) {
      atomicAdd(loss, scale * v);
    } else {                                 // summed in 64 bits; behind the sum, how many blocks are done
      atomicAdd(sum, (double)scale * v);
      __threadfence();
      if (atomicAdd(reinterpret_cast<unsigned*>(sum + 1), 1u) == gridDim.x * gridDim.y - 1) *loss = (float)atomicAdd(sum, 0.);
    }
  }
}

// ---------------------------------------------------------------------------------------------
// Soft-target KD + CE, one block per row:
//   loss += w_ce * CE(s, label) [label >= 0] + w_kd * T^2 * KL(softmax(t/T) || softmax(s/T))
//   gs    = w_ce * (softmax(s) - onehot) + w_kd * T * (softmax(s/T) - softmax(t/T))
// rows with row_mask == 0 are skipped (gradient zero).  `t` may be null when w_kd == 0.
//
// Two sweeps over the row.  The first keeps a running maximum and rescaled sums per thread (one rescale at most per 8
// elements), so the row leaves DRAM once; the second reads it again from L2 (148 SMs x 2 resident rows of 122 KB are
// 36 MB) and writes the gradient past L2's reuse order.  The sum that only cross-entropy needs is formed on labelled
// rows alone.  Bound by DRAM and, next to it, by the exponentials (four per element and two more on labelled rows).
// VEC: rows whose length is a multiple of 8 on 16-byte aligned bases are read and written 8 elements at a time.
// 8192 rows of 30528 bf16, one in seven labelled: 476 us (3.2 TB/s); three sweeps of single elements took 1810 us.
// ---------------------------------------------------------------------------------------------
struct RowPart {          // running maximum (-inf while empty)
  float m;
  __device__ __forceinline__ float ref() const { return fmaxf(m, -3.402823466e38f); }      // never -inf: exp(x - ref) is no NaN
};

// N values reduced over the block, the result in every thread; one barrier, so `sm` ([N][32]) is not used twice.
template <int N, bool MAX>
__device__ __forceinline__ void block_all(float (&v)[N], float* sm) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
#pragma unroll
  for (int k = 0; k < N; ++k) {
    v[k] = MAX ? tsp::warp_max(v[k]) : tsp::warp_sum(v[k]);
    if (lane == 0) sm[k * 32 + warp] = v[k];
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < N; ++k) {
    const float t = lane < nwarp ? sm[k * 32 + lane] : (MAX ? -INFINITY : 0.f);
    v[k] = MAX ? tsp::warp_max(t) : tsp::warp_sum(t);
  }
}

__device__ __forceinline__ float ex2(float x) {      // 2^x by the hardware's approximation, subnormal results as zero
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
constexpr float kLog2e = 1.4426950408889634f, kLn2 = 0.6931471805599453f;

template <typename TS, typename TT, bool VEC>
__global__ void __launch_bounds__(512, 2) kd_ce_kernel(const TS* __restrict__ s, const TT* __restrict__ t,
                                                       const int64_t* __restrict__ labels,
                                                       const uint8_t* __restrict__ row_mask, int n, int c, float temp,
                                                       float w_ce, float w_kd, double* __restrict__ loss,
                                                       TS* __restrict__ gs) {
  constexpr int V = VEC ? 8 : 1;
  __shared__ float scratch[6 * 32];
  const int row = blockIdx.x;
  if (row >= n) return;
  const TS* sr = s + (int64_t)row * c;
  const TT* tr = t ? t + (int64_t)row * c : nullptr;
  TS* gr = gs ? gs + (int64_t)row * c : nullptr;
  const int nv = c / V;
  if (row_mask != nullptr && row_mask[row] == 0) {
    const float zero[V] = {};
    if (gr) for (int i = threadIdx.x; i < nv; i += blockDim.x) store_part<TS, V>(gr, i, zero);
    return;
  }
  const bool kd = (w_kd != 0.f) && tr != nullptr;
  const float k2 = kLog2e / temp;                    // exponents are kept in powers of two
  const int64_t label = labels ? labels[row] : -1;
  const bool has_ce = (w_ce != 0.f) && label >= 0 && label < c;
  RowPart ps = {-INFINITY}, pt = {-INFINITY};
  float z1 = 0.f, zs = 0.f, zt = 0.f;
  for (int i = threadIdx.x; i < nv; i += blockDim.x) {
    float a[V], b[V];
    load_part<TS, V>(sr, i, a);
    if (kd) load_part<TT, V>(tr, i, b);
    float top = a[0];
#pragma unroll
    for (int e = 1; e < V; ++e) top = fmaxf(top, a[e]);
    if (top > ps.m) {
      const float d = ps.ref() - top;
      if (has_ce) z1 *= ex2(d * kLog2e);
      zs *= ex2(d * k2);
      ps.m = top;
    }
    const float rs = ps.ref();
    if (kd) {
#pragma unroll
      for (int e = 0; e < V; ++e) zs += ex2((a[e] - rs) * k2);
    }
    if (has_ce) {
#pragma unroll
      for (int e = 0; e < V; ++e) z1 += ex2((a[e] - rs) * kLog2e);
    }
    if (kd) {
      top = b[0];
#pragma unroll
      for (int e = 1; e < V; ++e) top = fmaxf(top, b[e]);
      if (top > pt.m) {
        zt *= ex2((pt.ref() - top) * k2);
        pt.m = top;
      }
      const float rt = pt.ref();
#pragma unroll
      for (int e = 0; e < V; ++e) zt += ex2((b[e] - rt) * k2);
    }
  }
  float m2[2] = {ps.m, pt.m};
  block_all<2, true>(m2, scratch);
  const float ms = m2[0], mt = m2[1];
  float z[3] = {z1 * ex2((ps.ref() - ms) * kLog2e), zs * ex2((ps.ref() - ms) * k2), kd ? zt * ex2((pt.ref() - mt) * k2) : 0.f};
  block_all<3, false>(z, scratch + 64);
  const float l1 = has_ce ? log2f(z[0]) : 0.f, ls = kd ? log2f(z[1]) : 0.f, lt = kd ? log2f(z[2]) : 0.f;
  // The divergence is sum p (db - da) / T - (ln Zt - ln Zs) with db, da the logits below their row's maximum, not a sum of
  // differences of logarithms: a class that the type's lowest value switches off stays finite at every temperature (times
  // log2(e) / T it is -inf below T = 1.44), and the logarithms' own rounding does not enter.  A class that the teacher gives
  // no probability adds nothing, whatever the other factor is (a NaN is kept).
  float kl = 0.f;
  const float wt = w_kd * temp;
  for (int i = threadIdx.x; i < nv; i += blockDim.x) {
    float a[V], b[V], g[V];
    load_part<TS, V>(sr, i, a);
    if (kd) load_part<TT, V>(tr, i, b);
    if (kd) {
#pragma unroll
      for (int e = 0; e < V; ++e) {
        const float da = a[e] - ms, db = b[e] - mt;
        const float p = ex2(db * k2 - lt);
        if (p != 0.f) kl = fmaf(p, db - da, kl);
        g[e] = wt * (ex2(da * k2 - ls) - p);
      }
    } else {
#pragma unroll
      for (int e = 0; e < V; ++e) g[e] = 0.f;
    }
    if (has_ce) {
#pragma unroll
      for (int e = 0; e < V; ++e) g[e] += w_ce * (ex2((a[e] - ms) * kLog2e - l1) - (i * V + e == (int)label ? 1.f : 0.f));
    }
    if (gr) store_part<TS, V>(gr, i, g);
  }
  float total[1] = {kl};
  if (kd) block_all<1, false>(total, scratch + 160);
  if (threadIdx.x == 0) {
    float v = 0.f;
    if (has_ce) v += w_ce * (l1 * kLn2 - (tsp::ld(sr, label) - ms));
    if (kd) v += w_kd * temp * (total[0] - temp * (lt - ls) * kLn2);
    atomicAdd(loss, (double)v);
  }
}

// out = in * gout, the scaling of a precomputed loss gradient by the gradient of the loss (a scalar in device memory),
// rounded to the tensor's type first as the product of two tensors of that type would be.  16-byte loads and stores, four in
// flight per thread.  In place (out == in) a factor of one leaves nothing to do: 500 MB of gradient, forward and backward of
// the loss above, 695 us with the pass and 531 without.
template <typename T> __device__ __forceinline__ float round_to(float v);
template <> __device__ __forceinline__ float round_to<float>(float v) { return v; }
template <> __device__ __forceinline__ float round_to<__nv_bfloat16>(float v) { return __bfloat162float(__float2bfloat16(v)); }

template <typename T>
__global__ void __launch_bounds__(256) scale_kernel(const T* in, const float* __restrict__ gout, T* out, int64_t n) {
  const float f = round_to<T>(*gout);
  if (in == out && f == 1.f) return;
  const int64_t nv = n >> 3, stride = (int64_t)gridDim.x * blockDim.x;
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t first = i;
  for (; i + 3 * stride < nv; i += 4 * stride) {
    tsp::Raw8<T> raw[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) tsp::ldraw(in, (i + u * stride) * 8, raw[u]);
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      float v[8];
      tsp::cvt8(raw[u], v);
#pragma unroll
      for (int e = 0; e < 8; ++e) v[e] *= f;
      tsp::st8(out, (i + u * stride) * 8, v);
    }
  }
  for (; i < nv; i += stride) {
    float v[8];
    tsp::ld8(in, i * 8, v);
#pragma unroll
    for (int e = 0; e < 8; ++e) v[e] *= f;
    tsp::st8(out, i * 8, v);
  }
  if (first < (n & 7)) tsp::st(out, (nv << 3) + first, tsp::ld(in, (nv << 3) + first) * f);
}

// ---------------------------------------------------------------------------------------------
// Cosine-embedding term of the DistilBERT loss (target +1): loss += scale * sum_rows (1 - cos) over selected rows
// ---------------------------------------------------------------------------------------------
template <typename T, bool VEC>
__global__ void __launch_bounds__(128) cosine_kernel(const T* __restrict__ x, const T* __restrict__ y,
                                                     const uint8_t* __restrict__ row_mask, int n, int d, float scale,
                                                     double* __restrict__ loss, T* __restrict__ gx) {
  constexpr int V = VEC ? 8 : 1;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int row = blockIdx.x * 4 + warp;
  const int nv = d / V;
  float contrib = 0.f;
  if (row < n) {
    const T* xr = x + (int64_t)row * d;
    const T* yr = y + (int64_t)row * d;
    T* gr = gx ? gx + (int64_t)row * d : nullptr;
    const bool on = row_mask == nullptr || row_mask[row] != 0;
    if (on) {
      float xx = 0.f, yy = 0.f, xy = 0.f;
      for (int i = lane; i < nv; i += 32) {
        float a[V], b[V];
        load_part<T, V>(xr, i, a);
        load_part<T, V>(yr, i, b);
#pragma unroll
        for (int e = 0; e < V; ++e) { xx += a[e] * a[e]; yy += b[e] * b[e]; xy += a[e] * b[e]; }
      }
      xx = tsp::warp_sum(xx) + 1e-8f; yy = tsp::warp_sum(yy) + 1e-8f; xy = tsp::warp_sum(xy);
      const float inv = rsqrtf(xx * yy);
      const float cosv = xy * inv;
      contrib = 1.f - cosv;
      if (gr) {
        const float c1 = -scale * inv, c2 = scale * cosv / xx;
        for (int i = lane; i < nv; i += 32) {
          float a[V], b[V];
          load_part<T, V>(xr, i, a);
          load_part<T, V>(yr, i, b);
#pragma unroll
          for (int e = 0; e < V; ++e) a[e] = c1 * b[e] + c2 * a[e];
          store_part<T, V>(gr, i, a);
        }
      }
    } else if (gr) {
      const float zero[V] = {};
      for (int i = lane; i < nv; i += 32) store_part<T, V>(gr, i, zero);
    }
  }
  __shared__ float part[4];
  if (lane == 0) part[warp] = contrib;
  __syncthreads();
  if (threadIdx.x == 0) atomicAdd(loss, (double)(scale * (part[0] + part[1] + part[2] + part[3])));
}

// The rows of a loss add to a 64-bit sum (`sum`, scratch): thousands of fp32 additions in turn are some 1e-6 off.
__global__ void round_sum_kernel(const double* __restrict__ sum, float* __restrict__ loss) { *loss = (float)*sum; }

// Rows of `d` elements on these bases can be accessed 8 elements (16 or 32 bytes) at a time.
bool rows_of_8(int d, const void* a, const void* b, const void* c) {
  return d % 8 == 0 && ((((uintptr_t)a) | ((uintptr_t)b) | ((uintptr_t)c)) & 15) == 0;
}

template <typename T>
int launch_byol(const void* x0, const void* y0, const void* x1, const void* y1, int n, int d, float scale, double* sum,
                float* loss, void* gx, cudaStream_t stream) {
  const PairPtrs<T> in = {{(const T*)x0, (const T*)x1}, {(const T*)y0, (const T*)y1}};
  const dim3 grid((n + 3) / 4, x1 != nullptr ? 2 : 1);
  const bool vec = rows_of_8(d, x0, y0, gx) && rows_of_8(d, x1, y1, nullptr);
  if (vec) byol_kernel<T, true><<<grid, 128, 0, stream>>>(in, n, d, scale, sum, loss, (T*)gx);
  else byol_kernel<T, false><<<grid, 128, 0, stream>>>(in, n, d, scale, sum, loss, (T*)gx);
  return TSP_LAUNCH_CHECK();
}

}  // namespace

extern "C" {

int tsp_byol_loss(const void* x, const void* y, int n, int d, int dtype, float scale, float* loss, void* gx,
                  cudaStream_t stream) {
  if (n <= 0) return 0;
  return dtype == TSP_DTYPE_BF16 ? launch_byol<__nv_bfloat16>(x, y, nullptr, nullptr, n, d, scale, nullptr, loss, gx, stream)
                                 : launch_byol<float>(x, y, nullptr, nullptr, n, d, scale, nullptr, loss, gx, stream);
}

// Both directions of the symmetric loss: loss = scale * sum of the pairs (x0, y0) and (x1, y1), set and not added to;
// gx [2][n][d]; `sum`: two doubles of scratch.
int tsp_byol_loss_pair(const void* x0, const void* y0, const void* x1, const void* y1, int n, int d, int dtype,
                       float scale, double* sum, float* loss, void* gx, cudaStream_t stream) {
  if (n <= 0) return (int)cudaMemsetAsync(loss, 0, sizeof(float), stream);
  cudaError_t e = cudaMemsetAsync(sum, 0, 2 * sizeof(double), stream);
  if (e != cudaSuccess) return (int)e;
  return dtype == TSP_DTYPE_BF16 ? launch_byol<__nv_bfloat16>(x0, y0, x1, y1, n, d, scale, sum, loss, gx, stream)
                                 : launch_byol<float>(x0, y0, x1, y1, n, d, scale, sum, loss, gx, stream);
}

int tsp_cosine_loss(const void* x, const void* y, const uint8_t* row_mask, int n, int d, int dtype, float scale,
                    double* sum, float* loss, void* gx, cudaStream_t stream) {
  if (n <= 0) return (int)cudaMemsetAsync(loss, 0, sizeof(float), stream);
  if (cudaError_t e = cudaMemsetAsync(sum, 0, sizeof(double), stream); e != cudaSuccess) return (int)e;
  const int grid = (n + 3) / 4;
  const bool vec = rows_of_8(d, x, y, gx);
#define TSP_COS(T, VEC) \
  cosine_kernel<T, VEC><<<grid, 128, 0, stream>>>((const T*)x, (const T*)y, row_mask, n, d, scale, sum, (T*)gx)
  if (dtype == TSP_DTYPE_BF16) { if (vec) TSP_COS(__nv_bfloat16, true); else TSP_COS(__nv_bfloat16, false); }
  else { if (vec) TSP_COS(float, true); else TSP_COS(float, false); }
#undef TSP_COS
  round_sum_kernel<<<1, 1, 0, stream>>>(sum, loss);
  return TSP_LAUNCH_CHECK();
}

int tsp_kd_ce_loss(const void* s, const void* t, const int64_t* labels, const uint8_t* row_mask, int n, int c,
                   int s_dtype, int t_dtype, float temp, float w_ce, float w_kd, double* sum, float* loss, void* gs,
                   cudaStream_t stream) {
  if (n <= 0) return (int)cudaMemsetAsync(loss, 0, sizeof(float), stream);
  if (cudaError_t e = cudaMemsetAsync(sum, 0, sizeof(double), stream); e != cudaSuccess) return (int)e;
  const bool vec = rows_of_8(c, s, t, gs);
  // at least four accesses per thread and sweep on long rows, one warp of latency on short ones
  const int parts = vec ? c / 8 : c;
  const int threads = parts >= 2048 ? 512 : parts >= 512 ? 256 : parts >= 96 ? 128 : 64;
#define TSP_KD(TS, TT)                                                                                               \
  do {                                                                                                               \
    if (vec)                                                                                                         \
      kd_ce_kernel<TS, TT, true><<<n, threads, 0, stream>>>((const TS*)s, (const TT*)t, labels, row_mask, n, c, temp, \
                                                            w_ce, w_kd, sum, (TS*)gs);                               \
    else                                                                                                             \
      kd_ce_kernel<TS, TT, false><<<n, threads, 0, stream>>>((const TS*)s, (const TT*)t, labels, row_mask, n, c,     \
                                                             temp, w_ce, w_kd, sum, (TS*)gs);                        \
  } while (0)
  if (s_dtype == TSP_DTYPE_BF16 && t_dtype == TSP_DTYPE_BF16) TSP_KD(__nv_bfloat16, __nv_bfloat16);
  else if (s_dtype == TSP_DTYPE_BF16) TSP_KD(__nv_bfloat16, float);
  else if (t_dtype == TSP_DTYPE_BF16) TSP_KD(float, __nv_bfloat16);
  else TSP_KD(float, float);
#undef TSP_KD
  round_sum_kernel<<<1, 1, 0, stream>>>(sum, loss);
  return TSP_LAUNCH_CHECK();
}

// out = in * *gout (see scale_kernel; out may be in); `in` and `out` 16-byte aligned.
int tsp_scale(const void* in, const float* gout, void* out, int64_t n, int dtype, cudaStream_t stream) {
  if (n <= 0) return 0;
  if ((((uintptr_t)in | (uintptr_t)out) & 15) != 0) return -2;
  int64_t blocks = (n / 8 + 1023) / 1024;
  if (blocks > 148 * 8) blocks = 148 * 8;
  if (blocks < 1) blocks = 1;
  if (dtype == TSP_DTYPE_BF16)
    scale_kernel<__nv_bfloat16><<<(int)blocks, 256, 0, stream>>>((const __nv_bfloat16*)in, gout, (__nv_bfloat16*)out, n);
  else
    scale_kernel<float><<<(int)blocks, 256, 0, stream>>>((const float*)in, gout, (float*)out, n);
  return TSP_LAUNCH_CHECK();
}

}  // extern "C"

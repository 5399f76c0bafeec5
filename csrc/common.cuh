// Shared device helpers for the sm_100a kernels of tspipe_b200.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#define TSP_DTYPE_F32 0
#define TSP_DTYPE_BF16 1

namespace tsp {

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// Block-wide sum; every thread gets the result.  `scratch` holds >= 33 floats.
__device__ __forceinline__ float block_sum(float v, float* scratch) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = (blockDim.x + 31) >> 5;
  v = warp_sum(v);
  __syncthreads();
  if (lane == 0) scratch[warp] = v;
  __syncthreads();
  if (warp == 0) {
    float t = lane < nwarp ? scratch[lane] : 0.f;
    t = warp_sum(t);
    if (lane == 0) scratch[32] = t;
  }
  __syncthreads();
  return scratch[32];
}

__device__ __forceinline__ float block_max(float v, float* scratch) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = (blockDim.x + 31) >> 5;
  v = warp_max(v);
  __syncthreads();
  if (lane == 0) scratch[warp] = v;
  __syncthreads();
  if (warp == 0) {
    float t = lane < nwarp ? scratch[lane] : -INFINITY;
    t = warp_max(t);
    if (lane == 0) scratch[32] = t;
  }
  __syncthreads();
  return scratch[32];
}

template <typename T> __device__ __forceinline__ float ld(const T* p, int64_t i);
template <> __device__ __forceinline__ float ld<float>(const float* p, int64_t i) { return p[i]; }
template <> __device__ __forceinline__ float ld<__nv_bfloat16>(const __nv_bfloat16* p, int64_t i) {
  return __bfloat162float(p[i]);
}
template <typename T> __device__ __forceinline__ void st(T* p, int64_t i, float v);
template <> __device__ __forceinline__ void st<float>(float* p, int64_t i, float v) { p[i] = v; }
template <> __device__ __forceinline__ void st<__nv_bfloat16>(__nv_bfloat16* p, int64_t i, float v) {
  p[i] = __float2bfloat16(v);
}

// 8 consecutive elements <-> 8 floats with one 16-byte (bf16) or two 16-byte (fp32) accesses.
// `p + i` must be 16-byte aligned.
template <typename T> __device__ __forceinline__ void ld8(const T* p, int64_t i, float (&v)[8]);
template <> __device__ __forceinline__ void ld8<float>(const float* p, int64_t i, float (&v)[8]) {
  const float4 a = *reinterpret_cast<const float4*>(p + i), b = *reinterpret_cast<const float4*>(p + i + 4);
  v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}
template <> __device__ __forceinline__ void ld8<__nv_bfloat16>(const __nv_bfloat16* p, int64_t i, float (&v)[8]) {
  const uint4 raw = *reinterpret_cast<const uint4*>(p + i);
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
  for (int k = 0; k < 4; ++k) { const float2 f = __bfloat1622float2(h[k]); v[2 * k] = f.x; v[2 * k + 1] = f.y; }
}
template <typename T> __device__ __forceinline__ void st8(T* p, int64_t i, const float (&v)[8]);
template <> __device__ __forceinline__ void st8<float>(float* p, int64_t i, const float (&v)[8]) {
  *reinterpret_cast<float4*>(p + i) = make_float4(v[0], v[1], v[2], v[3]);
  *reinterpret_cast<float4*>(p + i + 4) = make_float4(v[4], v[5], v[6], v[7]);
}
template <> __device__ __forceinline__ void st8<__nv_bfloat16>(__nv_bfloat16* p, int64_t i, const float (&v)[8]) {
  uint4 raw;
  __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&raw);
#pragma unroll
  for (int k = 0; k < 4; ++k) h[k] = __floats2bfloat162_rn(v[2 * k], v[2 * k + 1]);
  *reinterpret_cast<uint4*>(p + i) = raw;
}

// Raw 8-element vectors: issue the loads first (few registers), convert when consumed.
template <typename T> struct Raw8;
template <> struct Raw8<float> { float4 a, b; };
template <> struct Raw8<__nv_bfloat16> { uint4 a; };
__device__ __forceinline__ void ldraw(const float* p, int64_t i, Raw8<float>& r) {
  r.a = *reinterpret_cast<const float4*>(p + i);
  r.b = *reinterpret_cast<const float4*>(p + i + 4);
}
__device__ __forceinline__ void ldraw(const __nv_bfloat16* p, int64_t i, Raw8<__nv_bfloat16>& r) {
  r.a = *reinterpret_cast<const uint4*>(p + i);
}
// the same where ONCE, with evict-first hints: what is not read again soon
template <bool ONCE>
__device__ __forceinline__ void ldraw(const float* p, int64_t i, Raw8<float>& r) {
  if constexpr (!ONCE) return ldraw(p, i, r);
  r.a = __ldcs(reinterpret_cast<const float4*>(p + i));
  r.b = __ldcs(reinterpret_cast<const float4*>(p + i + 4));
}
template <bool ONCE>
__device__ __forceinline__ void ldraw(const __nv_bfloat16* p, int64_t i, Raw8<__nv_bfloat16>& r) {
  if constexpr (!ONCE) return ldraw(p, i, r);
  r.a = __ldcs(reinterpret_cast<const uint4*>(p + i));
}
__device__ __forceinline__ void cvt8(const Raw8<float>& r, float (&v)[8]) {
  v[0] = r.a.x; v[1] = r.a.y; v[2] = r.a.z; v[3] = r.a.w; v[4] = r.b.x; v[5] = r.b.y; v[6] = r.b.z; v[7] = r.b.w;
}
__device__ __forceinline__ void cvt8(const Raw8<__nv_bfloat16>& r, float (&v)[8]) {
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&r.a);
#pragma unroll
  for (int k = 0; k < 4; ++k) { const float2 f = __bfloat1622float2(h[k]); v[2 * k] = f.x; v[2 * k + 1] = f.y; }
}

// Two fp32 values that one instruction works on; each half is rounded as the scalar operation rounds.
struct Pair {
  uint64_t v;
  __device__ __forceinline__ Pair() {}
  __device__ __forceinline__ Pair(float a, float b) { asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(a), "f"(b)); }
  __device__ __forceinline__ void split(float& a, float& b) const { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
};
__device__ __forceinline__ Pair operator+(Pair a, Pair b) {
  Pair r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ Pair operator-(Pair a, Pair b) {
  Pair r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ Pair operator*(Pair a, Pair b) {
  Pair r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ Pair fma2(Pair a, Pair b, Pair c) {
  Pair r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}
__device__ __forceinline__ float total(Pair x) {
  float a, b;
  x.split(a, b);
  return a + b;
}
// two bf16 values as they lie in memory
__device__ __forceinline__ Pair unpack2(uint32_t x) { return Pair(__uint_as_float(x << 16), __uint_as_float(x & 0xffff0000u)); }

// The values as T holds them.
template <typename T, int N>
__device__ __forceinline__ void round_as(float (&v)[N]) {
  if constexpr (sizeof(T) == 2) {
#pragma unroll
    for (int e = 0; e < N; ++e) v[e] = __bfloat162float(__float2bfloat16(v[e]));
  }
}

// Blocks of `threads` threads for an elementwise pass over nvec vectors, cpv of them per row: `per_thread` vectors per
// thread where that leaves at least `least` blocks, fewer per thread (down to one) on smaller tensors, at most `most`
// blocks; rounded up so that the grid stride is a multiple of a row, i.e. a thread meets one column of vectors only.
inline int row_stride_blocks(int64_t nvec, int cpv, int threads, int per_thread, int64_t least, int64_t most) {
  const int64_t one = (nvec + threads - 1) / threads;
  int64_t g = (nvec + (int64_t)threads * per_thread - 1) / ((int64_t)threads * per_thread);
  if (g < least) g = one < least ? one : least;
  if (g > most) g = most;
  if (g < 1) g = 1;
  int a = cpv, b = threads;
  while (b != 0) { const int r = a % b; a = b; b = r; }
  const int64_t unit = cpv / a;                 // blocks after which a row begins on a block boundary again
  return (int)((g + unit - 1) / unit * unit);
}

// Unsigned division of numbers below 2^31 by a constant of the launch: multiply-high and shift (Granlund and Montgomery).
struct FastDiv {
  uint32_t d, mul, shift;
  FastDiv(uint32_t div = 1) : d(div), mul(0), shift(0) {
    while ((1ull << shift) < d) ++shift;
    mul = (uint32_t)((((1ull << shift) - d) << 32) / d + 1);
  }
  __device__ __forceinline__ uint32_t div(uint32_t n) const { return (__umulhi(mul, n) + n) >> shift; }
  __device__ __forceinline__ uint32_t div(uint32_t n, uint32_t& rest) const {
    const uint32_t q = div(n);
    rest = n - q * d;
    return q;
  }
};

// Hyperparameters of an optimizer's parameter groups for one launch.  They change from step to step (learning rates, bias
// corrections), so they travel with the launch: a table in device memory would have to be copied before each step.  Few
// groups go by value; a table serves more of them.  What does not change is a code per segment: group << 1 | adapt.
constexpr int kHyperVals = 8, kHyperGroups = 32;
struct Hyper {                                // (filled in by the caller: optim/flat.py has the same layout)
  const int* seg_code;                        // device memory
  const float* table;                         // [groups][kHyperVals] in device memory, or null
  float by_value[kHyperGroups][kHyperVals];
  __device__ __forceinline__ const float* of(int code) const {
    return table != nullptr ? table + kHyperVals * (int64_t)(code >> 1) : by_value[code >> 1];
  }
};
}  // namespace tsp

// ---------------------------------------------------------------------------------------------------------------------
// Launches that overlap the end of the kernel before them (programmatic dependent launch): the grid may be placed when every
// block of that kernel has called let_next_start or left, and wait_for_previous returns when it is complete and its writes
// are visible.  For the kernels that put one block on an SM (convolutions, products): their setup, and
// the way to the first operand, then overlap the end of the kernel before.  A grid that fills the SMs with several blocks each
// does not start this way: placed while the first SMs get free, its blocks end up unevenly on them.  A residual block at
// 14 x 14, 64 images (three convolutions, three normalisations), B200: in a CUDA graph 74.8 us with plain launches, 71.4 with all
// six early, 70.3 with the convolutions early; in a stream 88.1, 74.3 and 78.1.  Every reader of global memory comes after
// wait_for_previous.  Kernels that wait for other ranks neither start early nor let the next one.
// ---------------------------------------------------------------------------------------------------------------------
namespace tsp {
__device__ __forceinline__ void wait_for_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void let_next_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
// A pointer to what the kernel before has written, for use after wait_for_previous: through a `const __restrict__` parameter
// the compiler may load what it takes for constant before the wait.
template <typename P>
__device__ __forceinline__ P* written(P* p) {
  asm volatile("" : "+l"(p)::"memory");
  return p;
}
inline cudaLaunchAttribute early_start() {
  cudaLaunchAttribute a = {};
  a.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  a.val.programmaticStreamSerializationAllowed = 1;
  return a;
}
template <typename... P, typename... A>
inline cudaError_t launch_early(void (*kern)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, A&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1] = {early_start()};
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, static_cast<P>(args)...);
}
}  // namespace tsp

extern int g_tsp_sm_reserve;          // defined in peer.cu
namespace tsp {
// SMs that a persistent kernel may fill: all but those reserved for communication kernels (tsp_set_sm_reserve).
inline cudaError_t usable_sms(int& n) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
  n = n - g_tsp_sm_reserve > 8 ? n - g_tsp_sm_reserve : 8;
  return e;
}
}  // namespace tsp

// Every launcher returns the cudaError_t of its launch as int (0 = ok).
#define TSP_LAUNCH_CHECK() ((int)cudaGetLastError())

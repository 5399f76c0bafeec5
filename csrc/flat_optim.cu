// Optimizer and momentum-teacher kernels over flat parameter buffers (sm_100a).
//
// Reference behaviour: LARS `benchmarks/byol/main.py:13-46` (= `benchmarks/moco-v3/moco/optimizer.py`),
// AdamW / SGD from torch.optim as used by `benchmarks/distilbert/distiller.py:150` and
// `benchmarks/soft_target/train_kd.py:209-213`, momentum update `benchmarks/byol/trainer.py:198-212`.
// The reference runs 6-10 elementwise launches and two norm reductions PER TENSOR; here a whole
// partition is one flat fp32 buffer cut into fixed-size chunks that never straddle a tensor, so a step
// is one launch (LARS on buffers that fit L2: two), bound by HBM (or NVLink for a peer source).
#include "common.cuh"
#include "tspipe_kernels.h"

namespace {

using tsp::Hyper;

constexpr int kThreads = 256;
constexpr int kStepThreads = 256, kStepBlocks = 4;      // of lars_step_kernel, blocks per SM
constexpr uint64_t kWaitNs = 2000000000ull;             // its waits give up after two seconds

// ---------------------------------------------------------------------------------------------
// EMA: t = m*t + (1-m)*s ; `s` may point into a peer GPU's memory (plain loads over NVLink).
// Optionally writes a bf16 shadow of the new teacher for bf16 compute copies.
// ---------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(kThreads) ema_kernel(float* __restrict__ t, const float* __restrict__ s, int64_t n,
                                                       float m, __nv_bfloat16* __restrict__ shadow) {
  const float om = 1.f - m;
  const int64_t n4 = n >> 2;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  float4* t4 = reinterpret_cast<float4*>(t);
  const float4* s4 = reinterpret_cast<const float4*>(s);
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n4; i += stride) {
    float4 a = t4[i];
    const float4 b = __ldg(s4 + i);
    a.x = m * a.x + om * b.x; a.y = m * a.y + om * b.y; a.z = m * a.z + om * b.z; a.w = m * a.w + om * b.w;
    t4[i] = a;
    if (shadow) {
      __nv_bfloat162* sh = reinterpret_cast<__nv_bfloat162*>(shadow) + 2 * i;
      sh[0] = __floats2bfloat162_rn(a.x, a.y);
      sh[1] = __floats2bfloat162_rn(a.z, a.w);
    }
  }
  for (int64_t i = (n4 << 2) + (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    const float a = m * t[i] + om * s[i];
    t[i] = a;
    if (shadow) shadow[i] = __float2bfloat16(a);
  }
}

// ---------------------------------------------------------------------------------------------
// chunked multi-tensor kernels.  chunk = (segment id, first element, length); segment = one tensor.
// ---------------------------------------------------------------------------------------------
struct ChunkView {
  int seg;
  int64_t begin;
  int len;
};

__device__ __forceinline__ ChunkView load_chunk(const int64_t* __restrict__ chunks, int c) {
  ChunkView v;
  v.seg = (int)chunks[3 * (int64_t)c];
  v.begin = chunks[3 * (int64_t)c + 1];
  v.len = (int)chunks[3 * (int64_t)c + 2];
  return v;
}

// How many 16-byte vectors of a chunk can be updated at once: all of its body when the chunk starts on a vector, every
// buffer does (`bits`: their addresses or-ed) and the teacher's end does not cut a vector; none otherwise.  AdamW over 86.6 M
// parameters with the EMA teacher, 3.1 GB: 700 us with 4-byte accesses, 495 (6.3 TB/s) with 16-byte ones.
__device__ __forceinline__ int vec4_body(const ChunkView& c, uintptr_t bits, bool has_t, int64_t teacher_n) {
  return ((c.begin & 3) == 0 && (bits & 15) == 0 && !(has_t && (teacher_n & 3) != 0)) ? c.len >> 2 : 0;
}

// sum p^2 and sum (grad_scale*g + wd*p)^2 of this thread's share of a chunk
__device__ __forceinline__ void lars_sums(const float* p, const float* __restrict__ g, const ChunkView& c, float grad_scale,
                                          float wd, float& sp, float& su) {
  sp = 0.f; su = 0.f;
  const int n4 = ((c.begin & 3) == 0) ? (c.len >> 2) : 0;
  const float4* p4 = reinterpret_cast<const float4*>(p + c.begin);
  const float4* g4 = reinterpret_cast<const float4*>(g + c.begin);
#pragma unroll 4
  for (int i = threadIdx.x; i < n4; i += blockDim.x) {
    const float4 a = p4[i], b = g4[i];
    float u;
    sp += a.x * a.x + a.y * a.y + a.z * a.z + a.w * a.w;
    u = grad_scale * b.x + wd * a.x; su += u * u;
    u = grad_scale * b.y + wd * a.y; su += u * u;
    u = grad_scale * b.z + wd * a.z; su += u * u;
    u = grad_scale * b.w + wd * a.w; su += u * u;
  }
  for (int i = (n4 << 2) + threadIdx.x; i < c.len; i += blockDim.x) {
    const float a = p[c.begin + i], u = grad_scale * g[c.begin + i] + wd * a;
    sp += a * a; su += u * u;
  }
}

// norms[2*seg] += sum p^2 ; norms[2*seg+1] += sum (grad_scale*g + wd*p)^2   (only segments with the adapt bit)
__global__ void __launch_bounds__(kThreads) lars_norms_kernel(const float* __restrict__ p, const float* __restrict__ g,
                                                              const int64_t* __restrict__ chunks,
                                                              const __grid_constant__ Hyper hyper, float grad_scale,
                                                              float* __restrict__ norms) {
  __shared__ float scratch[33];
  const ChunkView c = load_chunk(chunks, blockIdx.x);
  const int code = hyper.seg_code[c.seg];
  if ((code & 1) == 0) return;
  float sp, su;
  lars_sums(p, g, c, grad_scale, hyper.of(code)[1], sp, su);         // lr, wd, momentum, trust
  sp = tsp::block_sum(sp, scratch);
  su = tsp::block_sum(su, scratch);
  if (threadIdx.x == 0) {
    atomicAdd(norms + 2 * c.seg, sp);
    atomicAdd(norms + 2 * c.seg + 1, su);
  }
}

template <bool ONCE>
__device__ __forceinline__ float4 ld_once(const float4* at) {
  if constexpr (ONCE) return __ldcs(at);
  else return *at;
}
template <bool ONCE>
__device__ __forceinline__ void st_once(float4* at, float4 v) {
  if constexpr (ONCE) __stcs(at, v);
  else *at = v;
}

// LARS update of a chunk (+ optional fused momentum-teacher update for segments that have a local teacher copy):
//   dp = adapt ? q*(gs*g + wd*p) : gs*g ; mu = mom*mu + dp ; p -= lr*mu ; [t = m*t + (1-m)*p]
// ONCE: nothing of it is read again soon, so loads and stores carry evict-first hints.
template <bool ONCE>
__device__ __forceinline__ void lars_update(float* p, const float* __restrict__ g, float* __restrict__ mu,
                                            const ChunkView& c, const float* hp, float q, float wd_eff, float grad_scale,
                                            float* __restrict__ teacher, int64_t teacher_n, float ema_m) {
  const float lr = hp[0], mom = hp[2];
  const float om = 1.f - ema_m;
  const bool has_t = teacher != nullptr;
  // 16-byte vectors over the aligned body (segments start on 256-byte boundaries), scalars for the tail
  const int n4 = ((c.begin & 3) == 0) ? (c.len >> 2) : 0;
  float4* p4 = reinterpret_cast<float4*>(p + c.begin);
  const float4* g4 = reinterpret_cast<const float4*>(g + c.begin);
  float4* m4 = reinterpret_cast<float4*>(mu + c.begin);
  float4* t4 = has_t ? reinterpret_cast<float4*>(teacher + c.begin) : nullptr;
#pragma unroll 2
  for (int i = threadIdx.x; i < n4; i += blockDim.x) {
    float4 pv = ld_once<ONCE>(p4 + i), mv = ld_once<ONCE>(m4 + i);
    const float4 gv = ld_once<ONCE>(g4 + i);
    const bool t_ok = has_t && (c.begin + 4 * (int64_t)i + 3 < teacher_n);
    float4 tv = t_ok ? ld_once<ONCE>(t4 + i) : make_float4(0.f, 0.f, 0.f, 0.f);
#define TSP_LARS1(X)                                                   \
    {                                                                  \
      const float dp = q * (grad_scale * gv.X + wd_eff * pv.X);        \
      mv.X = mom * mv.X + dp;                                          \
      pv.X -= lr * mv.X;                                               \
      tv.X = ema_m * tv.X + om * pv.X;                                 \
    }
    TSP_LARS1(x) TSP_LARS1(y) TSP_LARS1(z) TSP_LARS1(w)
#undef TSP_LARS1
    st_once<ONCE>(p4 + i, pv);
    st_once<ONCE>(m4 + i, mv);
    if (t_ok) st_once<ONCE>(t4 + i, tv);
  }
  for (int i = (n4 << 2) + threadIdx.x; i < c.len; i += blockDim.x) {
    const int64_t k = c.begin + i;
    const float pv = p[k];
    const float dp = q * (grad_scale * g[k] + wd_eff * pv);
    const float m2 = mom * mu[k] + dp;
    mu[k] = m2;
    const float np = pv - lr * m2;
    p[k] = np;
    if (has_t && k < teacher_n) teacher[k] = ema_m * teacher[k] + om * np;
  }
}

// Trust ratio of a segment from the sums of its squares.
__device__ __forceinline__ float lars_ratio(float trust, float pp, float uu) {
  const float pn = sqrtf(pp), un = sqrtf(uu);
  return (pn > 0.f && un > 0.f) ? trust * pn / un : 1.f;
}

// The second of two launches, behind lars_norms_kernel (or the exchange of norms between replicas).
__global__ void __launch_bounds__(kThreads) lars_apply_kernel(float* __restrict__ p, const float* __restrict__ g,
                                                              float* __restrict__ mu,
                                                              const int64_t* __restrict__ chunks,
                                                              const __grid_constant__ Hyper hyper, float grad_scale,
                                                              const float* __restrict__ norms,
                                                              float* __restrict__ teacher, int64_t teacher_n,
                                                              float ema_m) {
  const ChunkView c = load_chunk(chunks, blockIdx.x);
  const int code = hyper.seg_code[c.seg];
  const float* hp = hyper.of(code);
  const bool adapt = (code & 1) != 0;
  const float q = adapt ? lars_ratio(hp[3], norms[2 * c.seg], norms[2 * c.seg + 1]) : 1.f;
  lars_update<false>(p, g, mu, c, hp, q, adapt ? hp[1] : 0.f, grad_scale, teacher, teacher_n, ema_m);
}

// Norms and updates in one launch, for buffers that do not fit L2: a chunk's update follows its norms at a distance that
// L2 holds, so that what L2 keeps of p and g leaves DRAM once.  `order` lists the work: every chunk twice (row = {segment << 1 | update, length,
// begin}), its norms and, some chunks after the last norms of its segment, its update.  Blocks draw rows by ticket, so a
// wait for a segment's norms is a wait for rows that blocks drew before and are working on: whatever the number of
// resident blocks, the earliest unfinished row never waits.  sync[0] = ticket, sync[1 + seg] = pieces of the segment whose
// norms are in, sync[1 + n_seg] = a wait ran out; `need` = pieces per segment.  After a wait that ran out the step still ends: the
// segment's ratio is NaN then, and with it what is left to update of the segment, and *status (host memory) is set, which the
// optimizer raises on.  Bound by DRAM (p, g, mu, t once in, p, mu, t once out: 5.0 TB/s of it; by the counters L2 keeps some two
// fifths of p and g until the update, the rest is read again).  A step
// over 25.6 M parameters with the teacher, microseconds: two launches 160, this one 144; without the teacher 127 and 109; 86 M
// 494 and 463; 6 M (96 MB) 42 and 40.  Pieces of 32 KB and four blocks of 256 threads per SM: with pieces of 64 KB 147, of 16
// KB 152; two blocks of 512 threads 149; three blocks of 256 159.
__global__ void __launch_bounds__(kStepThreads, kStepBlocks)
lars_step_kernel(float* p, const float* __restrict__ g, float* __restrict__ mu, const int4* __restrict__ order,
                 int n_items, const int* __restrict__ need, const __grid_constant__ Hyper hyper, float grad_scale, float* norms,
                 int* sync, int n_seg, float* __restrict__ teacher, int64_t teacher_n, float ema_m, int* __restrict__ status) {
  __shared__ float scratch[33];
  __shared__ int4 row;
  __shared__ float ratio;
  __shared__ int done;                              // no row left
  int* gave_up = sync + 1 + n_seg;
  int next = 0;
  if (threadIdx.x == 0) next = atomicAdd(sync, 1);
  for (;;) {
    if (threadIdx.x == 0) {
      done = next < n_items ? 0 : 1;
      if (next < n_items) {
        row = __ldg(order + next);
        next = atomicAdd(sync, 1);                  // the ticket after this one, under way while this row is worked on
      }
    }
    __syncthreads();
    if (done != 0) return;
    ChunkView c;
    c.seg = row.x >> 1;
    c.len = row.y;
    c.begin = (int64_t)(uint32_t)row.z | ((int64_t)row.w << 32);
    const bool update = (row.x & 1) != 0;
    const int code = __ldg(hyper.seg_code + c.seg);
    const float* hp = hyper.of(code);
    const bool adapt = (code & 1) != 0;
    if (!update) {
      if (adapt) {
        float sp, su;
        lars_sums(p, g, c, grad_scale, hp[1], sp, su);
        sp = tsp::block_sum(sp, scratch);
        su = tsp::block_sum(su, scratch);
        if (threadIdx.x == 0) {
          atomicAdd(norms + 2 * c.seg, sp);
          atomicAdd(norms + 2 * c.seg + 1, su);
          __threadfence();
          atomicAdd(sync + 1 + c.seg, 1);
        }
      }
    } else {
      if (adapt && threadIdx.x == 0) {
        const int want = __ldg(need + c.seg);
        bool in = true;
        uint64_t t0 = 0;
        for (int spin = 0; *((volatile int*)(sync + 1 + c.seg)) < want; ++spin) {
          if ((spin & 31) != 31) continue;
          uint64_t now;
          asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
          if (t0 == 0) t0 = now;
          const bool late = now - t0 > kWaitNs;
          if (late || *((volatile int*)gave_up) != 0) {
            if (late) {
              atomicExch(gave_up, 1);
              *((volatile int*)status) = 1;
              __threadfence_system();
            }
            in = false;
            break;
          }
        }
        __threadfence();
        ratio = in ? lars_ratio(hp[3], __ldcg(norms + 2 * c.seg), __ldcg(norms + 2 * c.seg + 1)) : __int_as_float(0x7fffffff);
      }
      __syncthreads();
      lars_update<true>(p, g, mu, c, hp, adapt ? ratio : 1.f, adapt ? hp[1] : 0.f, grad_scale, teacher, teacher_n, ema_m);
    }
    __syncthreads();                                // the row and the ratio are read before the next ones are written
  }
}

// AdamW (decoupled weight decay), hyper-parameters of a group: lr, beta1, beta2, eps, wd, bias1, bias2
__global__ void __launch_bounds__(kThreads) adamw_kernel(float* __restrict__ p, const float* __restrict__ g,
                                                         float* __restrict__ m, float* __restrict__ v,
                                                         const int64_t* __restrict__ chunks,
                                                         const __grid_constant__ Hyper hyper, float grad_scale,
                                                         float* __restrict__ teacher, int64_t teacher_n, float ema_m) {
  const ChunkView c = load_chunk(chunks, blockIdx.x);
  const float* hp = hyper.of(hyper.seg_code[c.seg]);
  const float lr = hp[0], b1 = hp[1], b2 = hp[2], eps = hp[3], wd = hp[4], bc1 = hp[5], bc2 = hp[6];
  const float om = 1.f - ema_m;
  const float step = lr / bc1;
  const float inv_sqrt_bc2 = rsqrtf(bc2);
  const bool has_t = teacher != nullptr;
  auto one = [&](float& pv, float gv, float& mv, float& vv, float& tv) {
    gv *= grad_scale;
    pv *= 1.f - lr * wd;
    mv = b1 * mv + (1.f - b1) * gv;
    vv = b2 * vv + (1.f - b2) * gv * gv;
    pv -= step * mv / (sqrtf(vv) * inv_sqrt_bc2 + eps);
    tv = ema_m * tv + om * pv;
  };
  // 16-byte vectors over the aligned body (up to five loads in flight per thread and trip), scalars for the tail
  const int n4 = vec4_body(c, (uintptr_t)p | (uintptr_t)g | (uintptr_t)m | (uintptr_t)v | (uintptr_t)teacher, has_t, teacher_n);
  float4* p4 = reinterpret_cast<float4*>(p + c.begin);
  const float4* g4 = reinterpret_cast<const float4*>(g + c.begin);
  float4* m4 = reinterpret_cast<float4*>(m + c.begin);
  float4* v4 = reinterpret_cast<float4*>(v + c.begin);
  float4* t4 = has_t ? reinterpret_cast<float4*>(teacher + c.begin) : nullptr;
  for (int i = threadIdx.x; i < n4; i += kThreads) {
    float4 pv = p4[i], mv = m4[i], vv = v4[i];
    const float4 gv = g4[i];
    const bool t_ok = has_t && (c.begin + 4 * (int64_t)i + 3 < teacher_n);
    float4 tv = t_ok ? t4[i] : make_float4(0.f, 0.f, 0.f, 0.f);
    one(pv.x, gv.x, mv.x, vv.x, tv.x);
    one(pv.y, gv.y, mv.y, vv.y, tv.y);
    one(pv.z, gv.z, mv.z, vv.z, tv.z);
    one(pv.w, gv.w, mv.w, vv.w, tv.w);
    p4[i] = pv;
    m4[i] = mv;
    v4[i] = vv;
    if (t_ok) t4[i] = tv;
  }
  for (int i = (n4 << 2) + threadIdx.x; i < c.len; i += kThreads) {
    const int64_t k = c.begin + i;
    const bool t_ok = has_t && k < teacher_n;
    float pv = p[k], mv = m[k], vv = v[k], tv = t_ok ? teacher[k] : 0.f;
    one(pv, g[k], mv, vv, tv);
    p[k] = pv;
    m[k] = mv;
    v[k] = vv;
    if (t_ok) teacher[k] = tv;
  }
}

// SGD with momentum / nesterov / L2 weight decay; of a group: lr, momentum, dampening, wd, nesterov, first_step
__global__ void __launch_bounds__(kThreads) sgd_kernel(float* __restrict__ p, const float* __restrict__ g,
                                                       float* __restrict__ buf, const int64_t* __restrict__ chunks,
                                                       const __grid_constant__ Hyper hyper, float grad_scale,
                                                       float* __restrict__ teacher, int64_t teacher_n, float ema_m) {
  const ChunkView c = load_chunk(chunks, blockIdx.x);
  const float* hp = hyper.of(hyper.seg_code[c.seg]);
  const float lr = hp[0], mom = hp[1], damp = hp[2], wd = hp[3];
  const bool nesterov = hp[4] != 0.f, first = hp[5] != 0.f;
  const float om = 1.f - ema_m;
  const bool has_t = teacher != nullptr, has_b = mom != 0.f;
  auto one = [&](float& pv, float gv, float& bv, float& tv) {
    float d = grad_scale * gv + wd * pv;
    if (has_b) {
      bv = first ? d : mom * bv + (1.f - damp) * d;
      d = nesterov ? d + mom * bv : bv;
    }
    pv -= lr * d;
    tv = ema_m * tv + om * pv;
  };
  const int n4 = vec4_body(c, (uintptr_t)p | (uintptr_t)g | (uintptr_t)buf | (uintptr_t)teacher, has_t, teacher_n);
  float4* p4 = reinterpret_cast<float4*>(p + c.begin);
  const float4* g4 = reinterpret_cast<const float4*>(g + c.begin);
  float4* b4 = reinterpret_cast<float4*>(buf + c.begin);
  float4* t4 = has_t ? reinterpret_cast<float4*>(teacher + c.begin) : nullptr;
#pragma unroll 2
  for (int i = threadIdx.x; i < n4; i += kThreads) {
    float4 pv = p4[i];
    const float4 gv = g4[i];
    const bool t_ok = has_t && (c.begin + 4 * (int64_t)i + 3 < teacher_n);
    float4 bv = has_b && !first ? b4[i] : make_float4(0.f, 0.f, 0.f, 0.f);
    float4 tv = t_ok ? t4[i] : make_float4(0.f, 0.f, 0.f, 0.f);
    one(pv.x, gv.x, bv.x, tv.x);
    one(pv.y, gv.y, bv.y, tv.y);
    one(pv.z, gv.z, bv.z, tv.z);
    one(pv.w, gv.w, bv.w, tv.w);
    p4[i] = pv;
    if (has_b) b4[i] = bv;
    if (t_ok) t4[i] = tv;
  }
  for (int i = (n4 << 2) + threadIdx.x; i < c.len; i += kThreads) {
    const int64_t k = c.begin + i;
    const bool t_ok = has_t && k < teacher_n;
    float pv = p[k], bv = has_b && !first ? buf[k] : 0.f, tv = t_ok ? teacher[k] : 0.f;
    one(pv, g[k], bv, tv);
    p[k] = pv;
    if (has_b) buf[k] = bv;
    if (t_ok) teacher[k] = tv;
  }
}

inline int ema_grid(int64_t n) {
  int64_t blocks = (n / 4 + kThreads - 1) / kThreads;
  const int64_t cap = 148 * 8;
  if (blocks > cap) blocks = cap;
  if (blocks < 1) blocks = 1;
  return (int)blocks;
}

}  // namespace

extern "C" {

int tsp_ema_update(float* teacher, const float* student, int64_t n, float momentum, void* bf16_shadow,
                   cudaStream_t stream) {
  if (n <= 0) return 0;
  if ((reinterpret_cast<uintptr_t>(teacher) | reinterpret_cast<uintptr_t>(student)) & 15) return -2;
  ema_kernel<<<ema_grid(n), kThreads, 0, stream>>>(teacher, student, n, momentum,
                                                  reinterpret_cast<__nv_bfloat16*>(bf16_shadow));
  return TSP_LAUNCH_CHECK();
}

int tsp_lars_step(float* p, const float* g, float* mu, const int64_t* chunks, int n_chunks, const void* hyper,
                  float grad_scale, float* norms, int n_seg, float* teacher, int64_t teacher_n, float ema_m,
                  cudaStream_t stream) {
  if (n_chunks <= 0) return 0;
  cudaError_t e = cudaMemsetAsync(norms, 0, sizeof(float) * 2 * (size_t)n_seg, stream);
  if (e != cudaSuccess) return (int)e;
  lars_norms_kernel<<<n_chunks, kThreads, 0, stream>>>(p, g, chunks, *(const Hyper*)hyper, grad_scale, norms);
  lars_apply_kernel<<<n_chunks, kThreads, 0, stream>>>(p, g, mu, chunks, *(const Hyper*)hyper, grad_scale, norms, teacher,
                                                       teacher_n, ema_m);
  return TSP_LAUNCH_CHECK();
}

int tsp_lars_step_ordered(float* p, const float* g, float* mu, const void* order, int n_items, const int* need,
                          const void* hyper, float grad_scale, float* work, int n_seg, float* teacher, int64_t teacher_n,
                          float ema_m, int* status, cudaStream_t stream) {
  if (n_items <= 0) return 0;
  if ((reinterpret_cast<uintptr_t>(order) & 15) != 0) return -2;
  cudaError_t e = cudaMemsetAsync(work, 0, sizeof(float) * (3 * (size_t)n_seg + 2), stream);
  int sms = 0;
  if (e == cudaSuccess) e = tsp::usable_sms(sms);
  if (e != cudaSuccess) return (int)e;
  // (blocks for a whole number of SMs fewer: as many SMs are empty, or four times as many have room for a quarter of theirs)
  const int grid = n_items < kStepBlocks * sms ? n_items : kStepBlocks * sms;
  lars_step_kernel<<<grid, kStepThreads, 0, stream>>>(p, g, mu, (const int4*)order, n_items, need, *(const Hyper*)hyper,
                                                      grad_scale, work, (int*)(work + 2 * (size_t)n_seg), n_seg, teacher, teacher_n,
                                                      ema_m, status);
  return TSP_LAUNCH_CHECK();
}

int tsp_lars_norms(const float* p, const float* g, const int64_t* chunks, int n_chunks, const void* hyper,
                   float grad_scale, float* norms, int n_seg, cudaStream_t stream) {
  if (n_chunks <= 0) return 0;
  cudaError_t e = cudaMemsetAsync(norms, 0, sizeof(float) * 2 * (size_t)n_seg, stream);
  if (e != cudaSuccess) return (int)e;
  lars_norms_kernel<<<n_chunks, kThreads, 0, stream>>>(p, g, chunks, *(const Hyper*)hyper, grad_scale, norms);
  return TSP_LAUNCH_CHECK();
}

int tsp_lars_apply(float* p, const float* g, float* mu, const int64_t* chunks, int n_chunks, const void* hyper,
                   float grad_scale, const float* norms, float* teacher, int64_t teacher_n, float ema_m,
                   cudaStream_t stream) {
  if (n_chunks <= 0) return 0;
  lars_apply_kernel<<<n_chunks, kThreads, 0, stream>>>(p, g, mu, chunks, *(const Hyper*)hyper, grad_scale, norms, teacher,
                                                       teacher_n, ema_m);
  return TSP_LAUNCH_CHECK();
}

int tsp_adamw_step(float* p, const float* g, float* m, float* v, const int64_t* chunks, int n_chunks,
                   const void* hyper, float grad_scale, float* teacher, int64_t teacher_n, float ema_m,
                   cudaStream_t stream) {
  if (n_chunks <= 0) return 0;
  adamw_kernel<<<n_chunks, kThreads, 0, stream>>>(p, g, m, v, chunks, *(const Hyper*)hyper, grad_scale, teacher, teacher_n, ema_m);
  return TSP_LAUNCH_CHECK();
}

int tsp_sgd_step(float* p, const float* g, float* buf, const int64_t* chunks, int n_chunks, const void* hyper,
                 float grad_scale, float* teacher, int64_t teacher_n, float ema_m, cudaStream_t stream) {
  if (n_chunks <= 0) return 0;
  sgd_kernel<<<n_chunks, kThreads, 0, stream>>>(p, g, buf, chunks, *(const Hyper*)hyper, grad_scale, teacher, teacher_n, ema_m);
  return TSP_LAUNCH_CHECK();
}

}  // extern "C"

// Fused loss kernels (forward value + gradient in one launch), sm_100a.
//
// Reference math: BYOL regression `benchmarks/byol/trainer.py:51-55,192-196`; soft-target KD
// `benchmarks/soft_target/kd_losses/st.py:18-23` + CE `benchmarks/soft_target/train_kd.py:448-453`;
// DistilBERT KL/MLM-CE terms `benchmarks/distilbert/distiller.py:711-772`.  The reference evaluates each with
// 5-10 library ops (normalize, softmax, log_softmax, kl_div, cross_entropy, masked_select copies) and a
// second sweep in autograd; the loss GPU holds the whole mini-batch, so these are latency- and
// bandwidth-bound row kernels: one read of the rows (teacher rows may sit behind a peer pointer), one write of
// the student gradient.
#include "tcgen05.cuh"
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
// 8192 rows of 30528 bf16, one in seven labelled, none masked: 480 us (3.1 TB/s); three sweeps of single elements took 1810 us.
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

// ---------------------------------------------------------------------------------------------
// The same on long bf16 rows (a vocabulary), one persistent block per SM, one exponential per logit instead of two (three on
// labelled rows): the first sweep keeps e = 2^((x - m) k2), m a reference of the warp's, of the teacher in registers (one vector of
// five in shared memory) and of the student in shared memory (122 KB for 30528 classes), and the second only scales them by one
// factor per vector.  A reference is the maximum of the warp's first vectors until a vector is well above it.  The divergence is
// summed in the first sweep as well, sum e_t ((b - mt) - (a - ms)), and follows the references as the other sums do.  Meanwhile a
// producer warp streams the next rows into a ring with bulk copies.
// For rows that reach into the last vector, four of them per SM.  Microseconds with the kernel above and with this one, 15 in a
// hundred rows labelled, none masked: 8192 rows of 30528 classes 480 and 358, of 24584 398 and 323, 592 rows 53 and 45, 43 and 42;
// 300 rows, a quarter of them masked, 31 and 29, 26.5 and 27.8.
// What bounds it is the issue of instructions (270 per warp and vector of 8 pairs, 60 % of the slots) beside their latency: with
// all of the teacher's exponentials in registers, and the bounded wait unrolled with them, the registers of a block of 25 warps
// (72 a thread) did not do, and with 221 KB of shared memory in use what spills comes back from L2: 8192 rows as above 439.
// Fewer warps with more of a row each are slower for want of warps (12: 460 us where 24 took 410).
// Rows are drawn by ticket: masked ones cost next to nothing (the producer warp writes their zeros), so a fixed share of
// rows per block would leave blocks idle at the end.  Per row one barrier among the computing warps, behind the first
// sweep; its partial sums alternate between two buffers.
// ---------------------------------------------------------------------------------------------
constexpr int kRowWarps = 24, kRowThreads = kRowWarps * 32;     // computing threads; one more warp copies
constexpr int kRowVecs = 5;                                     // 16-byte vectors of a row per thread
constexpr int kPieceElems = kRowThreads * 8;                    // of one tensor: one vector per thread
constexpr int kPieceBytes = kPieceElems * 2;
constexpr int kRing = 3;                                        // pieces of s and t, 24 KB each
constexpr int kRowRegs = 4;                                     // vectors of the teacher's exponentials in registers
constexpr int kRowSmem = kRing * 2 * kPieceBytes + (2 * kRowVecs - kRowRegs) * kPieceElems * 4 + 2 * kRing * 8 + 128;
constexpr int kRowQueue = 4;                                    // rows that the ring and the sweeps may hold
static_assert(kRing < kRowQueue * 2 && kRowSmem <= 227 * 1024, "a row in the ring is two pieces at least");
constexpr uint64_t kRowWaitNs = 2000000000ull;                  // a wait gives up after two seconds
constexpr int kStreamMin = (kRowVecs - 1) * kPieceElems + 1;    // elements of a row: only the last vector is partly filled
constexpr int kStreamRows = 4;                                  // rows per SM that the kernel may use

using tsp::Pair;
using tsp::fma2;
using tsp::total;
using tsp::unpack2;
__device__ __forceinline__ Pair ex2(Pair x) {
  float a, b;
  x.split(a, b);
  return Pair(ex2(a), ex2(b));
}
// The largest of eight values as they lie in memory (NaN only where all are, as fmaxf).
__device__ __forceinline__ float top_of(const uint4& q) {
  auto h = [](uint32_t x) { return *reinterpret_cast<const __nv_bfloat162*>(&x); };
  const __nv_bfloat162 m = __hmax2(__hmax2(h(q.x), h(q.y)), __hmax2(h(q.z), h(q.w)));
  return fmaxf(__low2float(m), __high2float(m));
}
// sum e (d + shift) f from sum e d and z = sum e, where references move by `shift` and sums shrink by `f`; nothing is left
// of sums whose factor is zero, whatever they were
__device__ __forceinline__ float moved(float sum, float z, float f, float shift) {
  return f == 0.f ? 0.f : fmaf(z * f, shift, sum * f);
}
__device__ __forceinline__ float warp_top(float v) {            // as tsp::warp_max
  float r;
  asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
  return r;
}
// Sums of four values over the warp: of a in lanes 0 - 7, b in 8 - 15, c in 16 - 23, d in 24 - 31.
__device__ __forceinline__ float four_sums(float a, float b, float c, float d, int lane) {
  const bool h16 = (lane & 16) != 0, h8 = (lane & 8) != 0;
  const float x = (h16 ? c : a) + __shfl_xor_sync(0xffffffffu, h16 ? a : c, 16);
  const float y = (h16 ? d : b) + __shfl_xor_sync(0xffffffffu, h16 ? b : d, 16);
  float v = (h8 ? y : x) + __shfl_xor_sync(0xffffffffu, h8 ? x : y, 8);
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
// (a call: five copies of the bounded loop in the sweep cost registers that its values need)
__device__ __noinline__ bool wait_for_piece(uint64_t* bar, uint32_t phase, int* status) {
  return tc5::mbar_wait(bar, phase, status, 9, kRowWaitNs);
}
__device__ __forceinline__ void row_barrier() { asm volatile("bar.sync 1, %0;" ::"n"(kRowThreads) : "memory"); }

__global__ void __launch_bounds__(kRowThreads + 32, 1)
kd_ce_stream_kernel(const __nv_bfloat16* __restrict__ s, const __nv_bfloat16* __restrict__ t,
                    const int64_t* __restrict__ labels, const uint8_t* __restrict__ row_mask, int n, int c, float temp,
                    float w_ce, float w_kd, double* __restrict__ sum, float* __restrict__ loss,
                    __nv_bfloat16* __restrict__ gs) {
  extern __shared__ __align__(128) uint8_t ring[];
  float4* kept = (float4*)(ring + kRing * 2 * kPieceBytes);       // the student's exponentials, [vector][half][thread]
  uint64_t* full = (uint64_t*)(ring + kRing * 2 * kPieceBytes + (2 * kRowVecs - kRowRegs) * kPieceElems * 4);
  uint64_t* empty = full + kRing;
  __shared__ int2 rows[kRowQueue];                    // the rows in the ring: index (-1: no more) and label (-1: none)
  __shared__ float part[2][6][32];
  __shared__ int failed[2];                           // by row, as `part`: a wait of a computing warp ran out
  __shared__ double block_part;                       // the block's share of the loss
  __shared__ float2 refs[kRowWarps][kRowVecs];        // what a warp's exponentials refer to (see above), of s and t
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nv = c / 8;
  unsigned* counters = reinterpret_cast<unsigned*>(sum + 1);      // [0] ticket, [1] blocks that are done
  int* status = reinterpret_cast<int*>(sum + 2);      // not 0 once a wait has run out: the loss is NaN then
  if (threadIdx.x == 0) {
    for (int i = 0; i < kRing; ++i) {
      tc5::mbar_init(full + i, 1);
      tc5::mbar_init(empty + i, kRowWarps);
    }
    failed[0] = failed[1] = 0;
    block_part = 0.;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  if (warp == kRowWarps) {
    // ---------------- producer ----------------
    uint32_t it = 0;
    bool ok = true;
    for (int r = 0; ok;) {
      int row = 0;
      if (lane == 0) row = (int)atomicAdd(counters, 1u);
      row = __shfl_sync(0xffffffffu, row, 0);
      if (row < n && row_mask != nullptr && row_mask[row] == 0) {
        if (gs != nullptr) {
          uint4* gr = reinterpret_cast<uint4*>(gs + (int64_t)row * c);
          for (int i = lane; i < nv; i += 32) __stcs(gr + i, make_uint4(0, 0, 0, 0));
        }
        continue;
      }
      if (lane == 0) {
        int label = -1;
        if (row < n && labels != nullptr) {
          const int64_t l = labels[row];
          if (w_ce != 0.f && l >= 0 && l < c) label = (int)l;
        }
        for (int k = 0; k < kRowVecs && ok; ++k, ++it) {
          const int slot = it % kRing;
          const uint32_t round = it / kRing;
          if (round > 0) ok = tc5::mbar_wait_parked(empty + slot, (round - 1) & 1, status, 8, kRowWaitNs);
          if (!ok) break;
          // an entry is written again four rows on, behind a piece that every computing warp has released since it read it
          if (k == 0) rows[r % kRowQueue] = make_int2(row < n ? row : -1, label);
          if (row >= n) {
            tc5::mbar_arrive(full + slot);
            break;
          }
          const int first = k * kPieceElems;
          const int64_t at = (int64_t)row * c + first;
          const uint32_t bytes = 2u * (uint32_t)min(kPieceElems, c - first);
          uint8_t* dst = ring + slot * 2 * kPieceBytes;
          tc5::mbar_expect_tx(full + slot, 2 * bytes);
#pragma unroll
          for (int j = 0; j < 2; ++j)
            asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                             tc5::smem_u32(dst + j * kPieceBytes)),
                         "l"((j == 0 ? s : t) + at), "r"(bytes), "r"(tc5::smem_u32(full + slot))
                         : "memory");
        }
        if (row >= n) ok = false;
      }
      ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
      ++r;
    }
  } else {
    // ---------------- sweeps ----------------
    const float k2 = kLog2e / temp, wt = w_kd * temp;
    const Pair k2p(k2, k2);
    const float far = fminf(4.f, 4.f / k2);             // exponents stay below 4, and 6 without temperature: as exact as the exponentials
    uint32_t slot = 0, phase = 0;                       // of the next piece
    for (int r = 0;; ++r) {
      int2 id = make_int2(0, -1);
      bool ok = true;
      Pair et[kRowRegs][4];                             // the teacher's exponentials
      RowPart ps = {-INFINITY}, pt = {-INFINITY};
      float z1 = 0.f, zs = 0.f, zt = 0.f, kl = 0.f;
#pragma unroll
      for (int k = 0; k < kRowVecs; ++k) {
        // (a wait that ran out: the sums mean nothing then, and are used for nothing behind the barrier)
        if (!tc5::mbar_try_wait(tc5::smem_u32(full + slot), phase)) ok &= wait_for_piece(full + slot, phase, status);
        if (k == 0) id = rows[r % kRowQueue];
        if (k == 0 && id.x < 0) break;
        const uint4* piece = reinterpret_cast<const uint4*>(ring + slot * 2 * kPieceBytes) + threadIdx.x;
        const bool mine = k < kRowVecs - 1 || k * kRowThreads + (int)threadIdx.x < nv;
        uint4 qa = make_uint4(0, 0, 0, 0), qb = qa;
        if (mine) { qa = piece[0]; qb = piece[kPieceBytes / 16]; }
        __syncwarp();
        if (lane == 0) tc5::mbar_arrive(empty + slot);             // every lane has its vectors
        if (++slot == kRing) { slot = 0; phase ^= 1; }
        const float tops = warp_top(mine ? top_of(qa) : -INFINITY), topt = warp_top(mine ? top_of(qb) : -INFINITY);
        if (k == 0 || tops > ps.m + far || topt > pt.m + far) {
          const RowPart ns = {fmaxf(ps.m, tops)}, nt = {fmaxf(pt.m, topt)};
          const float ft = ex2((pt.ref() - nt.ref()) * k2);
          if (id.y >= 0) z1 *= ex2((ps.ref() - ns.ref()) * kLog2e);
          zs *= ex2((ps.ref() - ns.ref()) * k2);
          kl = moved(kl, zt, ft, (pt.ref() - ps.ref()) - (nt.ref() - ns.ref()));
          zt *= ft;
          ps = ns;
          pt = nt;
        }
        if (lane == 0) refs[warp][k] = make_float2(ps.ref(), pt.ref());
        if (mine) {
          const uint32_t a[4] = {qa.x, qa.y, qa.z, qa.w}, b[4] = {qb.x, qb.y, qb.z, qb.w};
          const Pair ms2(ps.ref(), ps.ref()), mt2(pt.ref(), pt.ref());
          Pair ss(0.f, 0.f), st(0.f, 0.f), sk(0.f, 0.f);
          float4* keep = kept + 2 * k * kRowThreads + threadIdx.x;
          Pair ek[4];                               // the teacher's
          float es[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const Pair da = unpack2(a[j]) - ms2, db = unpack2(b[j]) - mt2, ea = ex2(da * k2p);
            ek[j] = ex2(db * k2p);
            ss = ss + ea;
            st = st + ek[j];
            ea.split(es[2 * (j & 1)], es[2 * (j & 1) + 1]);
            if (j & 1) keep[(j >> 1) * kRowThreads] = make_float4(es[0], es[1], es[2], es[3]);
            sk = fma2(ek[j], db - da, sk);
          }
          if (id.y >= 0) {
            const Pair e2(kLog2e, kLog2e);
            Pair s1(0.f, 0.f);
#pragma unroll
            for (int j = 0; j < 4; ++j) s1 = s1 + ex2((unpack2(a[j]) - ms2) * e2);
            z1 += total(s1);
          }
          zs += total(ss);
          zt += total(st);
          float part_kl = total(sk);
          if (part_kl != part_kl) {                 // a class that the teacher gives no probability adds nothing, whatever
            part_kl = 0.f;                          // the other factor is
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              float p[2], d[2];
              ek[j].split(p[0], p[1]);
              ((unpack2(b[j]) - mt2) - (unpack2(a[j]) - ms2)).split(d[0], d[1]);
              part_kl = fmaf(p[1], p[1] != 0.f ? d[1] : 0.f, fmaf(p[0], p[0] != 0.f ? d[0] : 0.f, part_kl));
            }
          }
          kl += part_kl;
          if (k < kRowRegs) {
#pragma unroll
            for (int j = 0; j < 4; ++j) et[k < kRowRegs ? k : 0][j] = ek[j];
          } else {                                  // behind the student's
            float4* kt = keep + 2 * (kRowVecs - kRowRegs) * kRowThreads;
            float v[8];
#pragma unroll
            for (int j = 0; j < 4; ++j) ek[j].split(v[2 * j], v[2 * j + 1]);
            kt[0] = make_float4(v[0], v[1], v[2], v[3]);
            kt[kRowThreads] = make_float4(v[4], v[5], v[6], v[7]);
          }
        }
      }
      const bool has_ce = id.y >= 0;
      // the warp's sums, then the block's; a warp whose part is empty refers to a finite maximum
      float (*pp)[32] = part[r & 1];
      {
        const float v = four_sums(z1, zs, zt, kl, lane);
        if ((lane & 7) == 0) pp[2 + (lane >> 3)][warp] = v;
        if (lane == 0) { pp[0][warp] = ps.m; pp[1][warp] = pt.m; }
        if (!ok) *((volatile int*)(failed + (r & 1))) = 1;
      }
      row_barrier();
      if (*((volatile int*)(failed + (r & 1))) != 0 || id.x < 0) break;      // the same for all computing warps
      const bool in = lane < kRowWarps;
      const RowPart ws = {in ? pp[0][lane] : -INFINITY}, wtop = {in ? pp[1][lane] : -INFINITY};
      const float ms = warp_top(ws.m), mt = warp_top(wtop.m);
      // The divergence.  Before a part refers to the row's maximum, a class that the student has switched off (the type's lowest
      // value, -inf) can take it past the largest float, or to infinity where the teacher's probability will be no float: a row
      // with such a part has its divergence formed from the probabilities, behind the second sweep.
      const float part_kl = in ? moved(pp[5][lane], pp[4][lane], ex2((wtop.ref() - mt) * k2), (wtop.ref() - ws.ref()) - (mt - ms)) : 0.f;
      const bool redo = __any_sync(0xffffffffu, !(fabsf(part_kl) < 1e30f)) != 0;       // the same for all computing warps
      {
        const float v = four_sums(has_ce && in ? pp[2][lane] * ex2((ws.ref() - ms) * kLog2e) : 0.f,
                                  in ? pp[3][lane] * ex2((ws.ref() - ms) * k2) : 0.f, in ? pp[4][lane] * ex2((wtop.ref() - mt) * k2) : 0.f,
                                  part_kl, lane);
        z1 = __shfl_sync(0xffffffffu, v, 0);
        zs = __shfl_sync(0xffffffffu, v, 8);
        zt = __shfl_sync(0xffffffffu, v, 16);
        kl = __shfl_sync(0xffffffffu, v, 24);
      }
      const float l1 = has_ce ? log2f(z1) : 0.f, ls = log2f(zs), lt = log2f(zt);
      if (threadIdx.x == 0) atomicAdd(&block_part, (redo ? 0. : (double)(wt * (kl / zt))) - (double)(w_kd * temp * (temp * (lt - ls) * kLn2)));
      // second sweep: the gradient
      uint4* gr = gs ? reinterpret_cast<uint4*>(gs + (int64_t)id.x * c) : nullptr;
      const uint4* sr = reinterpret_cast<const uint4*>(s + (int64_t)id.x * c);
#pragma unroll
      for (int k = 0; k < kRowVecs; ++k) {
        const int i = k * kRowThreads + threadIdx.x;
        if (k < kRowVecs - 1 || i < nv) {
          const float2 ref = refs[warp][k];
          const float fs = wt * ex2((ref.x - ms) * k2 - ls), ft = -wt * ex2((ref.y - mt) * k2 - lt);
          const Pair fs2(fs, fs), ft2(ft, ft);
          const float4* keep = kept + 2 * k * kRowThreads + threadIdx.x;
          const float4 e0 = keep[0], e1 = keep[kRowThreads];
          Pair ek[4];
          if (k < kRowRegs) {
#pragma unroll
            for (int j = 0; j < 4; ++j) ek[j] = et[k < kRowRegs ? k : 0][j];
          } else {
            const float4* kt = keep + 2 * (kRowVecs - kRowRegs) * kRowThreads;
            const float4 t0 = kt[0], t1 = kt[kRowThreads];
            ek[0] = Pair(t0.x, t0.y);
            ek[1] = Pair(t0.z, t0.w);
            ek[2] = Pair(t1.x, t1.y);
            ek[3] = Pair(t1.z, t1.w);
          }
          Pair g[4] = {fma2(fs2, Pair(e0.x, e0.y), ft2 * ek[0]), fma2(fs2, Pair(e0.z, e0.w), ft2 * ek[1]),
                       fma2(fs2, Pair(e1.x, e1.y), ft2 * ek[2]), fma2(fs2, Pair(e1.z, e1.w), ft2 * ek[3])};
          float v[8];
#pragma unroll
          for (int j = 0; j < 4; ++j) g[j].split(v[2 * j], v[2 * j + 1]);
          if (has_ce) {                                 // (the row once more, from L2)
            const uint4 q = __ldg(sr + i);
            const uint32_t w[4] = {q.x, q.y, q.z, q.w};
            const Pair ms2(ms, ms), e2(kLog2e, kLog2e), minus_l2(-l1, -l1), wc(w_ce, w_ce);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const Pair d = unpack2(w[j]) - ms2;
              Pair p = ex2(fma2(d, e2, minus_l2));
              if (i * 4 + j == (id.y >> 1)) {
                float d0, d1;
                d.split(d0, d1);
                atomicAdd(&block_part, (double)(w_ce * (l1 * kLn2 - ((id.y & 1) ? d1 : d0))));
                p = p - ((id.y & 1) ? Pair(0.f, 1.f) : Pair(1.f, 0.f));
              }
              fma2(wc, p, g[j]).split(v[2 * j], v[2 * j + 1]);
            }
          }
          if (gr) __stcs(gr + i, make_uint4(tc5::pack_bf16x2(v[0], v[1]), tc5::pack_bf16x2(v[2], v[3]),
                                            tc5::pack_bf16x2(v[4], v[5]), tc5::pack_bf16x2(v[6], v[7])));
        }
      }
      if (redo) {                                       // as kd_ce_kernel forms it; the rows once more, from L2
        const uint4* tr = reinterpret_cast<const uint4*>(t + (int64_t)id.x * c);
        float part = 0.f;
#pragma unroll 1
        for (int i = threadIdx.x; i < nv; i += kRowThreads) {
          const uint4 qa = __ldg(sr + i), qb = __ldg(tr + i);
          const uint32_t a[4] = {qa.x, qa.y, qa.z, qa.w}, b[4] = {qb.x, qb.y, qb.z, qb.w};
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            float av[2], bv[2];
            unpack2(a[j]).split(av[0], av[1]);
            unpack2(b[j]).split(bv[0], bv[1]);
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              const float db = bv[e] - mt, p = ex2(db * k2 - lt);
              if (p != 0.f) part = fmaf(p, db - (av[e] - ms), part);
            }
          }
        }
        double wide = part;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) wide += __shfl_xor_sync(0xffffffffu, wide, o);
        if (lane == 0) atomicAdd(&block_part, (double)wt * wide);
      }
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    atomicAdd(sum, block_part);
    __threadfence();
    if (atomicAdd(counters + 1, 1u) == gridDim.x - 1)
      *loss = *((volatile int*)status) == 0 ? (float)atomicAdd(sum, 0.) : __int_as_float(0x7fffffff);
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

static void launch_cosine(const void* x, const void* y, const uint8_t* row_mask, int n, int d, int dtype, float scale,
                          double* sum, void* gx, cudaStream_t stream) {
  const int grid = (n + 3) / 4;
  const bool vec = rows_of_8(d, x, y, gx);
#define TSP_COS(T, VEC) \
  cosine_kernel<T, VEC><<<grid, 128, 0, stream>>>((const T*)x, (const T*)y, row_mask, n, d, scale, sum, (T*)gx)
  if (dtype == TSP_DTYPE_BF16) { if (vec) TSP_COS(__nv_bfloat16, true); else TSP_COS(__nv_bfloat16, false); }
  else { if (vec) TSP_COS(float, true); else TSP_COS(float, false); }
#undef TSP_COS
}

int tsp_cosine_loss(const void* x, const void* y, const uint8_t* row_mask, int n, int d, int dtype, float scale,
                    double* sum, float* loss, void* gx, cudaStream_t stream) {
  if (n <= 0) return (int)cudaMemsetAsync(loss, 0, sizeof(float), stream);
  if (cudaError_t e = cudaMemsetAsync(sum, 0, sizeof(double), stream); e != cudaSuccess) return (int)e;
  launch_cosine(x, y, row_mask, n, d, dtype, scale, sum, gx, stream);
  round_sum_kernel<<<1, 1, 0, stream>>>(sum, loss);
  return TSP_LAUNCH_CHECK();
}

// The loss of tsp_kd_ce_loss, on top of what *sum holds.
static int launch_kd_ce(const void* s, const void* t, const int64_t* labels, const uint8_t* row_mask, int n, int c,
                        int s_dtype, int t_dtype, float temp, float w_ce, float w_kd, double* sum, float* loss, void* gs,
                        cudaStream_t stream) {
  const bool vec = rows_of_8(c, s, t, gs);
  if (vec && t != nullptr && w_kd != 0.f && s_dtype == TSP_DTYPE_BF16 && t_dtype == TSP_DTYPE_BF16 &&
      c >= kStreamMin && c <= kRowVecs * kPieceElems) {
    int sms = 0;
    if (cudaError_t e = tsp::usable_sms(sms); e != cudaSuccess) return (int)e;
    if (n >= kStreamRows * sms) {
      cudaError_t e = cudaFuncSetAttribute(kd_ce_stream_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kRowSmem);
      if (e != cudaSuccess) return (int)e;
      kd_ce_stream_kernel<<<sms, kRowThreads + 32, kRowSmem, stream>>>(
          (const __nv_bfloat16*)s, (const __nv_bfloat16*)t, labels, row_mask, n, c, temp, w_ce, w_kd, sum, loss,
          (__nv_bfloat16*)gs);
      return TSP_LAUNCH_CHECK();
    }
  }
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

// `sum`: three doubles of scratch.
int tsp_kd_ce_loss(const void* s, const void* t, const int64_t* labels, const uint8_t* row_mask, int n, int c,
                   int s_dtype, int t_dtype, float temp, float w_ce, float w_kd, double* sum, float* loss, void* gs,
                   cudaStream_t stream) {
  if (n <= 0) return (int)cudaMemsetAsync(loss, 0, sizeof(float), stream);
  if (cudaError_t e = cudaMemsetAsync(sum, 0, 3 * sizeof(double), stream); e != cudaSuccess) return (int)e;
  return launch_kd_ce(s, t, labels, row_mask, n, c, s_dtype, t_dtype, temp, w_ce, w_kd, sum, loss, gs, stream);
}

// tsp_kd_ce_loss and tsp_cosine_loss over the same n rows and mask as one loss: the terms share the sum.
int tsp_distil_loss(const void* s, const void* t, const int64_t* labels, const uint8_t* row_mask, int n, int c,
                    int s_dtype, int t_dtype, float temp, float w_ce, float w_kd, const void* x, const void* y, int d,
                    int x_dtype, float scale, double* sum, float* loss, void* gs, void* gx, cudaStream_t stream) {
  if (n <= 0) return (int)cudaMemsetAsync(loss, 0, sizeof(float), stream);
  if (cudaError_t e = cudaMemsetAsync(sum, 0, 3 * sizeof(double), stream); e != cudaSuccess) return (int)e;
  launch_cosine(x, y, row_mask, n, d, x_dtype, scale, sum, gx, stream);
  if (const int rc = TSP_LAUNCH_CHECK(); rc != 0) return rc;
  return launch_kd_ce(s, t, labels, row_mask, n, c, s_dtype, t_dtype, temp, w_ce, w_kd, sum, loss, gs, stream);
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

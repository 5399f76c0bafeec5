// Microbatch BatchNorm for channels-last activations, fused with ReLU and the residual add (sm_100a).
//
// Reference: `tspipe/batchnorm.py:45-120` - F.batch_norm on the microbatch plus two extra full reductions
// (`input.sum`, `(input**2).sum`) for the deferred running statistics, followed by separate ReLU and
// residual-add kernels in the ResNet blocks (`benchmarks/byol/models/resnet_base_network.py`).  On B200 those
// memory-bound passes take more time than the convolutions.  Here:
//   forward  = statistics pass (per-channel sum / sum of squares; these ARE the deferred accumulators)
//              + one pass y = relu(scale*x + shift [+ residual]);
//   backward = reduction pass (sum dy', sum dy'*xhat with dy' = dy masked by y > 0; writes dy' as the residual
//              gradient when there is a residual) + one pass for dx.
// x is viewed as [M, C] with C contiguous (NHWC or [N, C]); C % 8 == 0; statistics in fp32.
#include "common.cuh"
#include "tspipe_kernels.h"

namespace {

constexpr int kBlock = 256;

// ---------------------------------------------------------------------------------------------
// per-channel sums:  out[c] += sum_rows a(r,c),  out[C + c] += sum_rows b(r,c)
//   MODE 0 (forward statistics): a = x, b = x*x
//   MODE 1 (backward reduction): a = dy', b = dy' * (x - mean) * rstd with dy' = dy masked by the ReLU:
//          mask from y > 0 when `y` is given (residual case), else recomputed as scale*x + shift > 0 when
//          `relu` is set (no extra tensor read); optionally stores dy' to dres.
//   MODE 2 (bias gradients): a = x, no b
//
// For what the streaming kernel below does not take: fp32, widths that are no power of two, tensors of at most a
// megabyte or so.  Those are bound by latency, so a block is 32 channel vectors (512 contiguous bytes of a row) by 8
// rows, every thread has 4 or 8 rows in flight, and the rows are split over as many blocks as fill the chip - down to
// one trip per thread.  The backward reduction of [2 x 128, 4096] bf16 and the bias gradients of 12608 rows (768 - 3072 columns, each), B200:
// 17.4 and 20 us with fewer rows in flight and additions that share sectors, 4.2 and 8 this way.
// grid = (row blocks, channel slabs, segments).
// ---------------------------------------------------------------------------------------------
struct Tile {
  int tx_n;   // threads along the channel-vector axis
  int ty_n;   // rows processed in parallel by a block
};

__host__ __device__ inline Tile make_tile(int cpv) {
  Tile t;
  t.tx_n = cpv < 32 ? cpv : 32;
  t.ty_n = kBlock / t.tx_n;
  return t;
}

template <typename T, int MODE> struct ColsumRows { static constexpr int value = MODE == 1 ? (sizeof(T) == 2 ? 3 : 2) : (sizeof(T) == 2 ? 8 : 4); };

template <typename T, int MODE>
__global__ void __launch_bounds__(kBlock, 2) bn_colsum_kernel(const T* __restrict__ x, const T* __restrict__ dy,
                                                           const T* __restrict__ y, T* __restrict__ dres,
                                                           const float* __restrict__ mean_rstd,
                                                           const float* __restrict__ w, const float* __restrict__ bias,
                                                           int relu, int64_t m, int c, float* __restrict__ out) {
  tsp::let_next_start();
  __shared__ float sm[(kBlock + 4) * 16];
  if constexpr (MODE == 2) {     // blockIdx.z = one of up to three matrices (x, dy, y), whose sums lie side by side
    if (blockIdx.z != 0) x = blockIdx.z == 1 ? dy : y;
    out += (int64_t)blockIdx.z * c;
  } else {   // blockIdx.z = segment: an independent group of m rows with its own statistics
    const int64_t so = (int64_t)blockIdx.z * m * c;
    x += so;
    if (dy != nullptr) dy += so;
    if (y != nullptr) y += so;
    if (dres != nullptr) dres += so;
    if (mean_rstd != nullptr) mean_rstd += (int64_t)blockIdx.z * 2 * c;
    out += (int64_t)blockIdx.z * 2 * c;
  }
  constexpr int U = ColsumRows<T, MODE>::value;
  const int cpv = c >> 3;
  const Tile tl = make_tile(cpv);
  const int tx = threadIdx.x % tl.tx_n, ty = threadIdx.x / tl.tx_n;
  const int cg = blockIdx.y * tl.tx_n + tx;
  const bool active = (ty < tl.ty_n) && (cg < cpv);
  float a[8], b[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) { a[e] = 0.f; b[e] = 0.f; }
  if (active) {
    // each block owns one contiguous range of rows
    const int64_t rows_per_block = (m + gridDim.x - 1) / gridDim.x;
    const int64_t r_begin = (int64_t)blockIdx.x * rows_per_block;
    const int64_t r_end = r_begin + rows_per_block < m ? r_begin + rows_per_block : m;
    const int64_t step = tl.ty_n, col = (int64_t)cg * 8;
    float mu[8], rs[8], sc[8], sh[8];
    const bool recompute_mask = (MODE == 1) && relu && (y == nullptr);
    if (MODE == 1) {
      tsp::ld8(mean_rstd, col, mu);
      tsp::ld8(mean_rstd + c, col, rs);
      if (recompute_mask) {
        float wv[8], bv[8];
        tsp::ld8(w, col, wv);
        tsp::ld8(bias, col, bv);
#pragma unroll
        for (int e = 0; e < 8; ++e) { sc[e] = wv[e] * rs[e]; sh[e] = bv[e] - mu[e] * sc[e]; }
      }
    }
    for (int64_t r = r_begin + ty; r < r_end; r += U * step) {
      // the loads of a trip are all issued before the first use; rows past the end are skipped
      tsp::Raw8<T> xr[U], gr[MODE == 1 ? U : 1], yr[MODE == 1 ? U : 1];
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (r + u * step < r_end) {
          const int64_t off = (r + u * step) * c + col;
          tsp::ldraw(x, off, xr[u]);
          if constexpr (MODE == 1) {
            tsp::ldraw(dy, off, gr[u]);
            if (y != nullptr) tsp::ldraw(y, off, yr[u]);
          }
        }
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (r + u * step < r_end) {
          float v[8];
          tsp::cvt8(xr[u], v);
          if constexpr (MODE == 0) {
#pragma unroll
            for (int e = 0; e < 8; ++e) { a[e] += v[e]; b[e] += v[e] * v[e]; }
          } else if constexpr (MODE == 2) {
#pragma unroll
            for (int e = 0; e < 8; ++e) a[e] += v[e];
          } else {
            float g[8];
            tsp::cvt8(gr[u], g);
            if (y != nullptr) {
              float yv[8];
              tsp::cvt8(yr[u], yv);
#pragma unroll
              for (int e = 0; e < 8; ++e) g[e] = yv[e] > 0.f ? g[e] : 0.f;
            } else if (recompute_mask) {
#pragma unroll
              for (int e = 0; e < 8; ++e) g[e] = (v[e] * sc[e] + sh[e]) > 0.f ? g[e] : 0.f;
            }
            if (dres != nullptr) tsp::st8(dres, (r + u * step) * c + col, g);
#pragma unroll
            for (int e = 0; e < 8; ++e) { a[e] += g[e]; b[e] += g[e] * (v[e] - mu[e]) * rs[e]; }
          }
        }
    }
  }
  // sum over ty through shared memory, then one addition per channel and block, lane = channel: a warp's additions go out
  // as whole sectors.  (Additions to one sector are serialised at some 15 ns each; with eight lanes' worth of
  // instructions per sector that was the whole time of the kernel.)
  constexpr int kVals = MODE == 2 ? 8 : 16;
  constexpr int pitch = kBlock + 4;                  // values 4 banks apart: the reads below are conflict-free
  if (ty < tl.ty_n) {
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      sm[e * pitch + threadIdx.x] = a[e];
      if (MODE != 2) sm[(8 + e) * pitch + threadIdx.x] = b[e];
    }
  }
  __syncthreads();
  for (int p = threadIdx.x; p < kVals * tl.tx_n; p += kBlock) {
    const int half = p >= 8 * tl.tx_n ? 1 : 0, q = p - half * 8 * tl.tx_n;
    const int e = q & 7, px = q >> 3, ch = blockIdx.y * tl.tx_n * 8 + q;
    if (ch < c) {
      float acc = 0.f;
      for (int k = 0; k < tl.ty_n; ++k) acc += sm[(half * 8 + e) * pitch + k * tl.tx_n + px];
      atomicAdd(out + half * c + ch, acc);
    }
  }
}

// ---------------------------------------------------------------------------------------------
// Streaming version of the per-channel sums for bf16 (same MODEs and results as bn_colsum_kernel).
//
// A read-only pass is bound by how many bytes an SM keeps in flight, not by arithmetic.  Instead of raising
// occupancy, one producer thread per CTA streams the CTA's contiguous row range through a ring of shared-memory
// buffers with bulk asynchronous copies (cp.async.bulk, completion on an mbarrier; 64 - 192 KB in flight per SM
// with no registers tied up), and 8 consumer warps read the buffers with conflict-free 16-byte loads.  With
// c/8 a power of two <= 256, consumer thread t always meets the channels 8 * (t % (c/8)) .. +7, so its partial
// sums stay in registers; one shared-memory reduction and one atomic per channel per CTA finish the job.
// Measured on [256*56*56, 256] bf16 (411 MB): 84 us = 4.9 TB/s, the same as a kernel that only reads.
//
// Waits are bounded (kStreamSpin polls); a wait that runs out sets g_bn_status and every role leaves its loop.
// ---------------------------------------------------------------------------------------------
constexpr int kStreamConsumers = 256;
constexpr int kStreamThreads = kStreamConsumers + 32;
constexpr int kStreamStages = 4;
constexpr uint32_t kStreamSpin = 1u << 22;
__device__ int g_bn_status = 0;

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ bool stream_wait(uint64_t* bar, uint32_t parity, int code) {
  const uint32_t addr = smem_u32(bar);
  for (uint32_t spin = 0; spin < kStreamSpin; ++spin) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.b32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(addr), "r"(parity)
        : "memory");
    if (done) return true;
    // The error word lives in global memory: the round trip to L2 per failed poll is the back-off of this loop
    // (polling flat out slowed the statistics pass from 38 us to 77 us on a 205 MB activation: the 8 waiting
    // warps took issue slots from the producer thread).
    if (*((volatile int*)&g_bn_status) != 0) return false;
  }
  atomicCAS(&g_bn_status, 0, code);
  return false;
}
__device__ __forceinline__ void stream_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}
__device__ __forceinline__ void unpack8(const uint4& raw, float (&v)[8]) {
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
  for (int k = 0; k < 4; ++k) { const float2 f = __bfloat1622float2(h[k]); v[2 * k] = f.x; v[2 * k + 1] = f.y; }
}

// NARR = number of streamed arrays: MODE 0: x; MODE 1: x, dy (, y).  `chunk` bytes per array and stage.
template <int MODE>
__global__ void __launch_bounds__(kStreamThreads, 1)
bn_colsum_stream_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ dy,
                        const __nv_bfloat16* __restrict__ y, __nv_bfloat16* __restrict__ dres,
                        const float* __restrict__ mean_rstd, const float* __restrict__ w,
                        const float* __restrict__ bias, int relu, int64_t m, int c, int chunk,
                        float* __restrict__ out) {
  extern __shared__ __align__(128) uint8_t stream_smem[];
  tsp::let_next_start();
  {   // blockIdx.y = segment: an independent group of m rows with its own statistics
    const int64_t so = (int64_t)blockIdx.y * m * c;
    x += so;
    if (dy != nullptr) dy += so;
    if (y != nullptr) y += so;
    if (dres != nullptr) dres += so;
    if (mean_rstd != nullptr) mean_rstd += (int64_t)blockIdx.y * 2 * c;
    out += (int64_t)blockIdx.y * 2 * c;
  }
  const int narr = MODE == 0 ? 1 : (y != nullptr ? 3 : 2);
  const int stage_bytes = narr * chunk;
  uint8_t* bufs = stream_smem;
  uint64_t* full = (uint64_t*)(stream_smem + kStreamStages * stage_bytes);
  uint64_t* empty = full + kStreamStages;
  float* red = (float*)(empty + kStreamStages);            // [kStreamConsumers][16]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int row_bytes = c * 2, cpv = c >> 3;
  const int rows_per_chunk = chunk / row_bytes;
  const int64_t rows_per_block = (m + gridDim.x - 1) / gridDim.x;
  const int64_t r_begin = (int64_t)blockIdx.x * rows_per_block;
  const int64_t r_end = r_begin + rows_per_block < m ? r_begin + rows_per_block : m;
  const int64_t nrows = r_end > r_begin ? r_end - r_begin : 0;
  const int n_chunks = (int)((nrows + rows_per_chunk - 1) / rows_per_chunk);
  if (tid == 0) {
    for (int s = 0; s < kStreamStages; ++s) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(full + s)), "r"(1));
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(empty + s)), "r"(kStreamConsumers / 32));
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  float a[8], b[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) { a[e] = 0.f; b[e] = 0.f; }
  if (warp == kStreamConsumers / 32) {
    // ---------------- producer ----------------
    if (lane == 0) {
      for (int i = 0; i < n_chunks; ++i) {
        const int s = i % kStreamStages;
        const uint32_t round = i / kStreamStages;
        if (round > 0 && !stream_wait(empty + s, (round - 1) & 1, 1)) break;
        const int64_t r0 = r_begin + (int64_t)i * rows_per_chunk;
        const int64_t rows = r_end - r0 < rows_per_chunk ? r_end - r0 : rows_per_chunk;
        const uint32_t bytes = (uint32_t)(rows * row_bytes);
        const int64_t off = r0 * row_bytes;
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(full + s)),
                     "r"(bytes * (uint32_t)narr)
                     : "memory");
        uint8_t* dst = bufs + s * stage_bytes;
        stream_load(dst, (const uint8_t*)x + off, bytes, full + s);
        if (MODE == 1) {
          stream_load(dst + chunk, (const uint8_t*)dy + off, bytes, full + s);
          if (narr == 3) stream_load(dst + 2 * chunk, (const uint8_t*)y + off, bytes, full + s);
        }
      }
    }
  } else {
    // ---------------- consumers ----------------
    const int cv = tid % cpv;                               // this thread's channel vector, fixed for all chunks
    float mu[8], rs[8], sc[8], sh[8];
    const bool recompute_mask = (MODE == 1) && relu && (y == nullptr);
    if (MODE == 1) {
      tsp::ld8(mean_rstd, (int64_t)cv * 8, mu);
      tsp::ld8(mean_rstd + c, (int64_t)cv * 8, rs);
      if (recompute_mask) {
        float wv[8], bv[8];
        tsp::ld8(w, (int64_t)cv * 8, wv);
        tsp::ld8(bias, (int64_t)cv * 8, bv);
#pragma unroll
        for (int e = 0; e < 8; ++e) { sc[e] = wv[e] * rs[e]; sh[e] = bv[e] - mu[e] * sc[e]; }
      }
    }
    for (int i = 0; i < n_chunks; ++i) {
      const int s = i % kStreamStages;
      const uint32_t round = i / kStreamStages;
      if (!stream_wait(full + s, round & 1, 2)) break;
      const int64_t r0 = r_begin + (int64_t)i * rows_per_chunk;
      const int64_t rows = r_end - r0 < rows_per_chunk ? r_end - r0 : rows_per_chunk;
      const int nvec = (int)(rows * cpv);
      const uint4* sx = (const uint4*)(bufs + s * stage_bytes);
      if (MODE == 0) {
        int v = tid;
        for (; v + 3 * kStreamConsumers < nvec; v += 4 * kStreamConsumers) {
          const uint4 q0 = sx[v], q1 = sx[v + kStreamConsumers], q2 = sx[v + 2 * kStreamConsumers],
                      q3 = sx[v + 3 * kStreamConsumers];
          float f[8];
          unpack8(q0, f);
#pragma unroll
          for (int e = 0; e < 8; ++e) { a[e] += f[e]; b[e] += f[e] * f[e]; }
          unpack8(q1, f);
#pragma unroll
          for (int e = 0; e < 8; ++e) { a[e] += f[e]; b[e] += f[e] * f[e]; }
          unpack8(q2, f);
#pragma unroll
          for (int e = 0; e < 8; ++e) { a[e] += f[e]; b[e] += f[e] * f[e]; }
          unpack8(q3, f);
#pragma unroll
          for (int e = 0; e < 8; ++e) { a[e] += f[e]; b[e] += f[e] * f[e]; }
        }
        for (; v < nvec; v += kStreamConsumers) {
          float f[8];
          unpack8(sx[v], f);
#pragma unroll
          for (int e = 0; e < 8; ++e) { a[e] += f[e]; b[e] += f[e] * f[e]; }
        }
      } else {
        const uint4* sg = (const uint4*)(bufs + s * stage_bytes + chunk);
        const uint4* sy = (const uint4*)(bufs + s * stage_bytes + 2 * chunk);
        uint4* gres = dres == nullptr ? nullptr : (uint4*)((uint8_t*)dres + r0 * row_bytes);
#pragma unroll 2
        for (int v = tid; v < nvec; v += kStreamConsumers) {
          float xv[8], g[8];
          unpack8(sx[v], xv);
          unpack8(sg[v], g);
          if (narr == 3) {
            float yv[8];
            unpack8(sy[v], yv);
#pragma unroll
            for (int e = 0; e < 8; ++e) g[e] = yv[e] > 0.f ? g[e] : 0.f;
          } else if (recompute_mask) {
#pragma unroll
            for (int e = 0; e < 8; ++e) g[e] = (xv[e] * sc[e] + sh[e]) > 0.f ? g[e] : 0.f;
          }
          if (gres != nullptr) {
            uint4 raw;
            __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&raw);
#pragma unroll
            for (int k = 0; k < 4; ++k) h[k] = __floats2bfloat162_rn(g[2 * k], g[2 * k + 1]);
            gres[v] = raw;
          }
#pragma unroll
          for (int e = 0; e < 8; ++e) { a[e] += g[e]; b[e] += g[e] * (xv[e] - mu[e]) * rs[e]; }
        }
      }
      __syncwarp();
      if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(empty + s)) : "memory");
    }
#pragma unroll
    for (int e = 0; e < 8; ++e) { red[tid * 16 + e] = a[e]; red[tid * 16 + 8 + e] = b[e]; }
  }
  if (*((volatile int*)&g_bn_status) != 0) {
    for (int i = 0; i < 64; ++i) __nanosleep(1000);        // let copies that are still in flight land
  }
  __syncthreads();
  // threads with equal tid % cpv hold the same channels: sum the groups, one atomic per channel and CTA
  const int groups = kStreamConsumers / cpv;
  for (int p = tid; p < 16 * cpv; p += kStreamThreads) {
    const int cv = p >> 4, e = p & 15;
    float acc = 0.f;
    for (int g = 0; g < groups; ++g) acc += red[(g * cpv + cv) * 16 + e];
    atomicAdd(out + (e < 8 ? 0 : c) + cv * 8 + (e & 7), acc);
  }
}

// ---------------------------------------------------------------------------------------------
// forward apply: y = act(scale*x + shift [+ res]).
//   training: mean/var from `sums` (sum, sum of squares over m rows); the first threads save mean / rstd and fold the
//             sums into the deferred accumulators (acc_sum, acc_sumsq) when given.
//   eval:     mean/var from `fixed` ([mean | var]).
// The grid stride is a multiple of c/8 (apply_blocks), so a thread meets one channel vector only and derives its scale
// and shift itself, in registers, while its first activations are on their way.  (A table of all channels per block,
// behind a barrier, cost more than the pass itself on the small tensors: [2 x 128, 4096] took 27.6 us with it and takes 8.0.)
// ---------------------------------------------------------------------------------------------
// vectors in flight per thread and array (64 - 80 registers)
template <typename T> struct ApplyVecs {
  static constexpr int fwd = sizeof(T) == 2 ? 4 : 2, fwd_res = sizeof(T) == 2 ? 3 : 1, bwd = sizeof(T) == 2 ? 2 : 1;
};

// Activations up to this size find room in the L2 cache (126 MB) for the next kernel, which is a convolution of them as a rule.  The pass
// then reads with evict-first hints, so that its output stays there and not the inputs.  ResNet-50 forward, B200: 32
// images 1228 us -> 1210, 64 1762 -> 1722, 96 2422 -> 2379, 128 3000 -> 2970.  The hints on larger activations: training bottlenecks
// of 205 and 411 MB 890 -> 894 and 1661 -> 1671; in the backward's pass, whose output meets two kernels that read as much again, no difference.
constexpr int64_t kStaysInL2 = 126 << 20;

// ONCE: x and res are read with evict-first hints
template <typename T, bool RES, bool ONCE>
__global__ void __launch_bounds__(kBlock, 3) bn_apply_kernel(const T* __restrict__ x, const T* __restrict__ res,
                                                          T* __restrict__ y, const float* __restrict__ sums,
                                                          const float* __restrict__ fixed,
                                                          const float* __restrict__ w, const float* __restrict__ b,
                                                          float* __restrict__ save_mean_rstd,
                                                          float* __restrict__ acc_sum, float* __restrict__ acc_sumsq,
                                                          float* __restrict__ acc_count, int64_t acc_seg_stride,
                                                          int64_t m, int c, float eps, int relu) {
  tsp::let_next_start();
  {   // blockIdx.y = segment: m rows with their own statistics (and their own set of accumulators)
    const int64_t so = (int64_t)blockIdx.y * m * c;
    x += so;
    y += so;
    if (RES) res += so;
    if (sums != nullptr) sums += (int64_t)blockIdx.y * 2 * c;
    if (save_mean_rstd != nullptr) save_mean_rstd += (int64_t)blockIdx.y * 2 * c;
    if (acc_sum != nullptr) { acc_sum += blockIdx.y * acc_seg_stride; acc_sumsq += blockIdx.y * acc_seg_stride; }
    if (acc_count != nullptr) acc_count += blockIdx.y * acc_seg_stride;
  }
  constexpr int U = RES ? ApplyVecs<T>::fwd_res : ApplyVecs<T>::fwd;
  const int cpv = c >> 3;
  const int64_t nvec = m * cpv;
  const int64_t stride = (int64_t)gridDim.x * kBlock;
  const int first = blockIdx.x * kBlock + threadIdx.x;
  int64_t i = first;
  if (i >= nvec) return;
  const int ch = (first % cpv) * 8;
  tsp::Raw8<T> xr[U], rr[RES ? U : 1];
  auto load = [&](int64_t at) {
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (at + u * stride < nvec) {
        tsp::ldraw<ONCE>(x, (at + u * stride) * 8, xr[u]);
        if constexpr (RES) tsp::ldraw<ONCE>(res, (at + u * stride) * 8, rr[u]);
      }
  };
  load(i);
  float sc[8], sh[8];
  {
    float mean[8], var[8];
    if (fixed != nullptr) {
      tsp::ld8(fixed, ch, mean);
      tsp::ld8(fixed + c, ch, var);
    } else {
      const float inv_m = 1.f / (float)m;
      float s[8], q[8];
      tsp::ld8(sums, ch, s);
      tsp::ld8(sums + c, ch, q);
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        mean[e] = s[e] * inv_m;
        var[e] = fmaxf(q[e] * inv_m - mean[e] * mean[e], 0.f);
      }
      if (first < cpv) {                                  // the first c/8 threads own the channels' bookkeeping
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          if (acc_sum != nullptr) { acc_sum[ch + e] += s[e]; acc_sumsq[ch + e] += q[e]; }
          if (acc_count != nullptr) acc_count[ch + e] += (float)m;
        }
      }
    }
    float wv[8], bv[8];
    if (w != nullptr) tsp::ld8(w, ch, wv);
    if (b != nullptr) tsp::ld8(b, ch, bv);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const float rstd = rsqrtf(var[e] + eps);
      if (first < cpv && save_mean_rstd != nullptr) { save_mean_rstd[ch + e] = mean[e]; save_mean_rstd[c + ch + e] = rstd; }
      sc[e] = (w != nullptr ? wv[e] : 1.f) * rstd;
      sh[e] = (b != nullptr ? bv[e] : 0.f) - mean[e] * sc[e];
    }
  }
  while (true) {
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (i + u * stride < nvec) {
        float o[8];
        tsp::cvt8(xr[u], o);
#pragma unroll
        for (int e = 0; e < 8; ++e) o[e] = o[e] * sc[e] + sh[e];
        if constexpr (RES) {
          float r[8];
          tsp::cvt8(rr[u], r);
#pragma unroll
          for (int e = 0; e < 8; ++e) o[e] += r[e];
        }
        if (relu) {
#pragma unroll
          for (int e = 0; e < 8; ++e) o[e] = fmaxf(o[e], 0.f);
        }
        tsp::st8(y, (i + u * stride) * 8, o);
      }
    i += U * stride;
    if (i >= nvec) break;
    load(i);
  }
}

// ---------------------------------------------------------------------------------------------
// backward apply: dx = w*rstd * (dy' - sum(dy')/m - xhat * sum(dy'*xhat)/m), dy' masked as in the reduction
// (by y > 0 when `y` is given, by scale*x + shift > 0 when `relu` is set and y is null).
// Per element: dx = A*dy' + B*x + D with A = w*rstd, B = -A*rstd*k2, D = -A*k1 - B*mean, in registers as above.
// ---------------------------------------------------------------------------------------------
// MASK: 0 none, 1 recomputed from x, 2 from y
template <typename T, int MASK>
__global__ void __launch_bounds__(kBlock, 3) bn_bwd_apply_kernel(const T* __restrict__ dy, const T* __restrict__ x,
                                                              const T* __restrict__ y,
                                                              const float* __restrict__ mean_rstd,
                                                              const float* __restrict__ w,
                                                              const float* __restrict__ bias,
                                                              const float* __restrict__ sums, T* __restrict__ dx,
                                                              float* __restrict__ gw, float* __restrict__ gb,
                                                              int64_t m, int c) {
  tsp::let_next_start();
  {   // blockIdx.y = segment
    const int64_t so = (int64_t)blockIdx.y * m * c;
    dy += so;
    x += so;
    dx += so;
    if (MASK == 2) y += so;
    mean_rstd += (int64_t)blockIdx.y * 2 * c;
    sums += (int64_t)blockIdx.y * 2 * c;
  }
  constexpr int U = ApplyVecs<T>::bwd;
  const int cpv = c >> 3;
  const int64_t nvec = m * cpv;
  const int64_t stride = (int64_t)gridDim.x * kBlock;
  const int first = blockIdx.x * kBlock + threadIdx.x;
  int64_t i = first;
  if (i >= nvec) return;
  const int ch = (first % cpv) * 8;
  tsp::Raw8<T> gr[U], xr[U], yr[MASK == 2 ? U : 1];
  auto load = [&](int64_t at) {
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (at + u * stride < nvec) {
        tsp::ldraw(dy, (at + u * stride) * 8, gr[u]);
        tsp::ldraw(x, (at + u * stride) * 8, xr[u]);
        if constexpr (MASK == 2) tsp::ldraw(y, (at + u * stride) * 8, yr[u]);
      }
  };
  load(i);
  if (gw != nullptr && blockIdx.y == 0 && first < cpv) {      // the parameters' gradients: the sums over the segments
    for (int e = 0; e < 8; ++e) {
      float db = 0.f, dw = 0.f;
      for (int g = 0; g < (int)gridDim.y; ++g) { db += sums[(int64_t)g * 2 * c + ch + e]; dw += sums[(int64_t)(g * 2 + 1) * c + ch + e]; }
      gb[ch + e] += db;
      gw[ch + e] += dw;
    }
  }
  float A[8], B[8], D[8], sh[8];
  {
    const float inv_m = 1.f / (float)m;
    float mean[8], rs[8], k1[8], k2[8], wv[8], bv[8];
    tsp::ld8(mean_rstd, ch, mean);
    tsp::ld8(mean_rstd + c, ch, rs);
    tsp::ld8(sums, ch, k1);
    tsp::ld8(sums + c, ch, k2);
    if (w != nullptr) tsp::ld8(w, ch, wv);
    if (bias != nullptr) tsp::ld8(bias, ch, bv);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      A[e] = (w != nullptr ? wv[e] : 1.f) * rs[e];
      B[e] = -A[e] * rs[e] * (k2[e] * inv_m);
      D[e] = -A[e] * (k1[e] * inv_m) - B[e] * mean[e];
      sh[e] = (bias != nullptr ? bv[e] : 0.f) - mean[e] * A[e];
    }
  }
  while (true) {
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (i + u * stride < nvec) {
        float g[8], xv[8], o[8];
        tsp::cvt8(gr[u], g);
        tsp::cvt8(xr[u], xv);
        if constexpr (MASK == 2) {
          float yv[8];
          tsp::cvt8(yr[u], yv);
#pragma unroll
          for (int e = 0; e < 8; ++e) g[e] = yv[e] > 0.f ? g[e] : 0.f;
        } else if constexpr (MASK == 1) {
#pragma unroll
          for (int e = 0; e < 8; ++e) g[e] = (xv[e] * A[e] + sh[e]) > 0.f ? g[e] : 0.f;
        }
#pragma unroll
        for (int e = 0; e < 8; ++e) o[e] = A[e] * g[e] + B[e] * xv[e] + D[e];
        tsp::st8(dx, (i + u * stride) * 8, o);
      }
    i += U * stride;
    if (i >= nvec) break;
    load(i);
  }
}

// ---------------------------------------------------------------------------------------------
// BatchNorm + ReLU + 3x3 / stride 2 / pad 1 max-pool (the ResNet stem) without the normalised activation in memory.
//
// The passes are bound by the arithmetic on every element of x as much as by memory, so two channels share an instruction
// wherever bf16 allows it (Duo).  Values are rounded to T before they are compared, so the result is that of the separate
// passes.
// Forward: a row's maximum over the three columns, and a window's over the three rows, with the winner's code and its element
// of x selected by the mask "the first one is the maximum".  A thread walks a strip of output rows of one column and 8 channels
// (an odd row is the last of one window and the first of the next) and has the next window's rows on their way meanwhile.  idx
// gets the winner's code, kNoTap where the maximum is zero: there the ReLU passes no gradient.
// Backward: the gradient meets the winners only, so the two sums need dy and the winners (an output-sized tensor instead of x),
// as the reduction of a BatchNorm + ReLU over them.  In the pass for dx, dy' of an input pixel is gathered from the <= 4 windows
// it belongs to, instead of being scattered to an activation-sized tensor.  A thread takes 2 x 2 blocks of input pixels, which
// meet exactly the four windows (a, b) .. (a + 1, b + 1), down a strip of rows, two channels at a time.
// A block is kBlock / (c / 8) pixels by all channels (by 2048 of them, blockIdx.z, where there are more).
// 128 images of 112 x 112 x 64 bf16 (205 MB), B200: forward for a backward 90 us with keys of value and code for each
// channel, without the winners' elements; 83 this way with them (51 MB more).  Without a backward (64 images) 46 and 32.  Backward:
// the sums 79 from x and 25 from the winners, dx 109 with a load of four windows per block and 87 this way (floor 75).
// ---------------------------------------------------------------------------------------------
// Codes of the taps, for two channels: a byte each, in the upper half of a 16-bit lane, where every code reads as a bf16 number
// that is no denormal but for zero, and no NaN: comparisons of bf16 pairs compare codes.
__host__ __device__ constexpr uint32_t lanes(uint32_t code) { return code << 8 | code << 24; }
constexpr uint32_t kNoTap = lanes(0xff);
__host__ __device__ constexpr uint32_t tap_code(int ky, int kx) { return lanes((uint32_t)((2 - ky) * 4 + 2 - kx)); }

using tsp::FastDiv;
struct PoolGeom {
  int n, h, w, c, ho, wo;      // images of one segment, extents
  int rows;                    // output rows of a strip, which a thread walks from top to bottom
  FastDiv by_wo, by_strips;    // by_strips: strips of an image
  uint32_t items;              // strips of one column each, of one segment
};

// Two neighbouring channels: values as T holds them, and masks to select by.
template <typename T> struct Duo;
template <> struct Duo<__nv_bfloat16> {
  using V = uint32_t;
  using M = uint32_t;
  static __device__ __forceinline__ __nv_bfloat162 h(V v) { return *reinterpret_cast<__nv_bfloat162*>(&v); }
  static __device__ __forceinline__ V u(__nv_bfloat162 v) { return *reinterpret_cast<uint32_t*>(&v); }
  static __device__ __forceinline__ V get(const tsp::Raw8<__nv_bfloat16>& r, int j) { return reinterpret_cast<const uint32_t*>(&r.a)[j]; }
  static __device__ __forceinline__ void set(tsp::Raw8<__nv_bfloat16>& r, int j, V v) { reinterpret_cast<uint32_t*>(&r.a)[j] = v; }
  static __device__ __forceinline__ tsp::Pair wide(V v) { return tsp::unpack2(v); }
  static __device__ __forceinline__ V round(tsp::Pair p) {
    float a, b;
    p.split(a, b);
    return u(__floats2bfloat162_rn(a, b));
  }
  static __device__ __forceinline__ V lowest() { return 0xff80ff80u; }
  static __device__ __forceinline__ V larger(V a, V b) { return u(__hmax2(h(a), h(b))); }
  static __device__ __forceinline__ V sum(V a, V b) { return u(__hadd2(h(a), h(b))); }
  static __device__ __forceinline__ M equal(V a, V b) { return __heq2_mask(h(a), h(b)); }
  static __device__ __forceinline__ M same_code(uint32_t a, uint32_t b) { return __heq2_mask(h(a), h(b)); }
  static __device__ __forceinline__ V pick(M m, V a, V b) { return (m & a) | (~m & b); }
  static __device__ __forceinline__ V keep(M m, V a) { return m & a; }
  static __device__ __forceinline__ uint32_t pick_code(M m, uint32_t a, uint32_t b) { return (m & a) | (~m & b); }
};
template <> struct Duo<float> {
  using V = float2;
  struct M { bool a, b; };
  static __device__ __forceinline__ V get(const tsp::Raw8<float>& r, int j) { return reinterpret_cast<const float2*>(&r)[j]; }
  static __device__ __forceinline__ void set(tsp::Raw8<float>& r, int j, V v) { reinterpret_cast<float2*>(&r)[j] = v; }
  static __device__ __forceinline__ tsp::Pair wide(V v) { return tsp::Pair(v.x, v.y); }
  static __device__ __forceinline__ V round(tsp::Pair p) {
    float2 v;
    p.split(v.x, v.y);
    return v;
  }
  static __device__ __forceinline__ V lowest() { return make_float2(-INFINITY, -INFINITY); }
  static __device__ __forceinline__ V larger(V a, V b) { return make_float2(fmaxf(a.x, b.x), fmaxf(a.y, b.y)); }
  static __device__ __forceinline__ V sum(V a, V b) { return make_float2(a.x + b.x, a.y + b.y); }
  static __device__ __forceinline__ M equal(V a, V b) { return {a.x == b.x, a.y == b.y}; }
  static __device__ __forceinline__ M same_code(uint32_t a, uint32_t b) { return {(a & 0xffffu) == (b & 0xffffu), (a >> 16) == (b >> 16)}; }
  static __device__ __forceinline__ V pick(M m, V a, V b) { return make_float2(m.a ? a.x : b.x, m.b ? a.y : b.y); }
  static __device__ __forceinline__ V keep(M m, V a) { return make_float2(m.a ? a.x : 0.f, m.b ? a.y : 0.f); }
  static __device__ __forceinline__ uint32_t pick_code(M m, uint32_t a, uint32_t b) {
    return __byte_perm(m.a ? a : b, m.b ? a : b, 0x7610);
  }
};
template <typename T>
__device__ __forceinline__ void st_raw(T* p, int64_t i, const tsp::Raw8<T>& r) {
  if constexpr (sizeof(T) == 2) {
    *reinterpret_cast<uint4*>(p + i) = r.a;
  } else {
    *reinterpret_cast<float4*>(p + i) = r.a;
    *reinterpret_cast<float4*>(p + i + 4) = r.b;
  }
}

// The channel vector and the first pixel of a thread, the pixels of a block.
struct PoolThread {
  int per_block, slot, vec;
  bool active;
  __device__ __forceinline__ explicit PoolThread(int cpv) {
    const int width = min(cpv, kBlock);
    per_block = kBlock / width;
    slot = threadIdx.x / width;
    vec = blockIdx.z * kBlock + threadIdx.x % width;
    active = slot < per_block && vec < cpv;
  }
};

// WIN: with idx and won, for the backward.
template <typename T, bool WIN>
__global__ void __launch_bounds__(kBlock, sizeof(T) == 2 ? 3 : 2) bn_relu_pool_kernel(const T* __restrict__ x, T* __restrict__ y,
                                                              uint8_t* __restrict__ idx, T* __restrict__ won,
                                                              const float* __restrict__ sums,
                                                              const float* __restrict__ wgt,
                                                              const float* __restrict__ bias,
                                                              float* __restrict__ save_mean_rstd,
                                                              float* __restrict__ acc_sum, float* __restrict__ acc_sumsq,
                                                              float* __restrict__ acc_count, int64_t acc_seg_stride,
                                                              const PoolGeom g, float eps) {
  tsp::let_next_start();
  using D = Duo<T>;
  using V = typename D::V;
  {   // blockIdx.y = segment
    const int64_t seg = blockIdx.y;
    x += seg * g.n * g.h * g.w * g.c;
    y += seg * g.n * g.ho * g.wo * g.c;
    if (WIN) { idx += seg * g.n * g.ho * g.wo * g.c; won += seg * g.n * g.ho * g.wo * g.c; }
    sums += seg * 2 * g.c;
    save_mean_rstd += seg * 2 * g.c;
    if (acc_sum != nullptr) { acc_sum += seg * acc_seg_stride; acc_sumsq += seg * acc_seg_stride; }
    if (acc_count != nullptr) acc_count += seg * acc_seg_stride;
  }
  const int c = g.c;
  const PoolThread th(c >> 3);
  if (!th.active) return;
  const int ch = th.vec * 8;
  tsp::Pair scale[4], shift[4];
  {
    float sc[8], sh[8];
    const float rows = (float)((int64_t)g.n * g.h * g.w), inv_m = 1.f / rows;
    float s[8], q[8], wv[8], bv[8];
    tsp::ld8(sums, ch, s);
    tsp::ld8(sums + c, ch, q);
    tsp::ld8(wgt, ch, wv);
    tsp::ld8(bias, ch, bv);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const float mean = s[e] * inv_m, rstd = rsqrtf(fmaxf(q[e] * inv_m - mean * mean, 0.f) + eps);
      if (blockIdx.x == 0 && th.slot == 0) {
        if (acc_sum != nullptr) { acc_sum[ch + e] += s[e]; acc_sumsq[ch + e] += q[e]; }
        if (acc_count != nullptr) acc_count[ch + e] += rows;
        save_mean_rstd[ch + e] = mean;
        save_mean_rstd[c + ch + e] = rstd;
      }
      sc[e] = wv[e] * rstd;
      sh[e] = bv[e] - mean * sc[e];
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      scale[j] = tsp::Pair(sc[2 * j], sc[2 * j + 1]);
      shift[j] = tsp::Pair(sh[2 * j], sh[2 * j + 1]);
    }
  }
  const int pitch = g.w * c;                     // (below 2^31: n * h * w is)
  for (uint32_t i = blockIdx.x * th.per_block + th.slot; i < g.items; i += gridDim.x * th.per_block) {
    const uint32_t strip = g.by_wo.div(i), img = g.by_strips.div(strip);
    const int ox = (int)(i - strip * g.by_wo.d), oy0 = (int)(strip - img * g.by_strips.d) * g.rows;
    const int end = min(oy0 + g.rows, g.ho);
    const bool left = ox > 0, right = 2 * ox + 1 < g.w;
    const T* xi = x + ((int64_t)img * g.h + 2 * oy0) * pitch + (2 * ox) * c + ch;      // the centre of the first window
    int64_t o = (((int64_t)img * g.ho + oy0) * g.wo + ox) * c + ch;
    auto load = [&](const T* row, tsp::Raw8<T> (&raw)[3]) {      // (a column that does not exist: any other)
      tsp::ldraw(row, left ? -c : 0, raw[0]);
      tsp::ldraw(row, 0, raw[1]);
      tsp::ldraw(row, right ? c : 0, raw[2]);
    };
    // The largest value of a row over the window's columns, or of some rows, the first of equal ones: its element of x, its code.
    struct Best { V v[4], raw[4]; uint32_t code[4]; };
    auto better = [&](V& v, V& raw, uint32_t& code, V v2, V raw2, uint32_t code2) {      // of this one and a later one
      const V m = D::larger(v, v2);
      if (WIN) {
        const auto first = D::equal(v, m);
        raw = D::pick(first, raw, raw2);
        code = D::pick_code(first, code, code2);
      }
      v = m;
    };
    auto of_row = [&](const tsp::Raw8<T> (&raw)[3], uint32_t row_code, Best& r) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        V v[3];
#pragma unroll
        for (int kx = 0; kx < 3; ++kx) v[kx] = D::round(tsp::fma2(D::wide(D::get(raw[kx], j)), scale[j], shift[j]));
        if (!left) v[0] = D::lowest();
        if (!right) v[2] = D::lowest();
        r.v[j] = v[0];
        r.raw[j] = D::get(raw[0], j);
        r.code[j] = row_code | lanes(2);
        better(r.v[j], r.raw[j], r.code[j], v[1], D::get(raw[1], j), row_code | lanes(1));
        better(r.v[j], r.raw[j], r.code[j], v[2], D::get(raw[2], j), row_code);
      }
    };
    tsp::Raw8<T> raw0[3], raw1[3];
    Best top;                                    // the row above the window's centre
    if (oy0 > 0) load(xi - pitch, raw1);
    load(xi, raw0);
    if (oy0 > 0) of_row(raw1, 0, top);
    if (2 * oy0 + 1 < g.h) load(xi + pitch, raw1);
#pragma unroll 1
    for (int oy = oy0; oy < end; ++oy) {
      Best mid, win;
      of_row(raw0, lanes(4), mid);
      if (oy + 1 < end) load(xi + 2 * (int64_t)pitch, raw0);     // on their way while this window is formed
      if (oy > 0) {
        win = top;
#pragma unroll
        for (int j = 0; j < 4; ++j) better(win.v[j], win.raw[j], win.code[j] |= lanes(8), mid.v[j], mid.raw[j], mid.code[j]);
      } else {
        win = mid;
      }
      if (2 * oy + 1 < g.h) {                    // (an odd height ends in a window of two rows)
        of_row(raw1, 0, top);
        if (oy + 1 < end && 2 * oy + 3 < g.h) load(xi + 3 * (int64_t)pitch, raw1);
#pragma unroll
        for (int j = 0; j < 4; ++j) better(win.v[j], win.raw[j], win.code[j], top.v[j], top.raw[j], top.code[j]);
      }
      tsp::Raw8<T> out, w;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const V zero = {}, v = D::larger(win.v[j], zero);
        D::set(out, j, v);
        if (WIN) {
          D::set(w, j, win.raw[j]);
          win.code[j] = D::pick_code(D::equal(v, zero), kNoTap, win.code[j]);
        }
      }
      st_raw(y, o, out);
      if (WIN) {
        st_raw(won, o, w);
        *reinterpret_cast<uint2*>(idx + o) = make_uint2(__byte_perm(win.code[0], win.code[1], 0x7531),
                                                        __byte_perm(win.code[2], win.code[3], 0x7531));
      }
      xi += 2 * (int64_t)pitch;
      o += (int64_t)g.wo * c;
    }
  }
}

// dx from the two sums of the gradient behind the ReLU (sums[seg], by the reduction over the winners).
template <typename T>
__global__ void __launch_bounds__(kBlock, 2) bn_relu_pool_bwd_kernel(const T* __restrict__ dy, const uint8_t* __restrict__ idx,
                                                                  const T* __restrict__ x,
                                                                  const float* __restrict__ mean_rstd,
                                                                  const float* __restrict__ wgt,
                                                                  const float* __restrict__ sums, T* __restrict__ dx,
                                                                  float* __restrict__ gw, float* __restrict__ gb,
                                                                  const PoolGeom g) {
  tsp::let_next_start();
  using D = Duo<T>;
  using V = typename D::V;
  const int c = g.c;
  {   // blockIdx.y = segment
    const int64_t seg = blockIdx.y, in = seg * g.n * g.h * g.w * c, outs = seg * g.n * g.ho * g.wo * c;
    x += in;
    dx += in;
    dy += outs;
    idx += outs;
    mean_rstd += seg * 2 * c;
    sums += seg * 2 * c;
  }
  const PoolThread th(c >> 3);
  const int ch = th.vec * 8;
  if (!th.active) return;
  if (gw != nullptr && blockIdx.y == 0 && blockIdx.x == 0 && th.slot == 0) {
    for (int e = 0; e < 8; ++e) {
      float db = 0.f, dw = 0.f;
      for (int k = 0; k < (int)gridDim.y; ++k) { db += sums[(int64_t)k * 2 * c + ch + e]; dw += sums[(int64_t)(k * 2 + 1) * c + ch + e]; }
      gb[ch + e] += db;
      gw[ch + e] += dw;
    }
  }
  tsp::Pair A[4], B[4], C[4];                   // dx = A dy' + B x + C
  {
    float mean[8], rs[8], wv[8], k1[8], k2[8];
    tsp::ld8(mean_rstd, ch, mean);
    tsp::ld8(mean_rstd + c, ch, rs);
    tsp::ld8(wgt, ch, wv);
    tsp::ld8(sums, ch, k1);
    tsp::ld8(sums + c, ch, k2);
    const float inv_m = 1.f / (float)((int64_t)g.n * g.h * g.w);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float a[2], b[2], d[2];
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        const int e = 2 * j + s;
        a[s] = wv[e] * rs[e];
        b[s] = -a[s] * rs[e] * (k2[e] * inv_m);
        d[s] = -a[s] * (k1[e] * inv_m) - b[s] * mean[e];
      }
      A[j] = tsp::Pair(a[0], a[1]);
      B[j] = tsp::Pair(b[0], b[1]);
      C[j] = tsp::Pair(d[0], d[1]);
    }
  }
  const int64_t out_pitch = (int64_t)g.wo * c, in_pitch = (int64_t)g.w * c;
  for (uint32_t i = blockIdx.x * th.per_block + th.slot; i < g.items; i += gridDim.x * th.per_block) {
    const uint32_t strip = g.by_wo.div(i), img = g.by_strips.div(strip);
    const int wb = (int)(i - strip * g.by_wo.d), wa0 = (int)(strip - img * g.by_strips.d) * g.rows;
    const int end = min(wa0 + g.rows, g.ho);
    const bool right = wb + 1 < g.wo, col1 = 2 * wb + 1 < g.w;          // the window to the right, the second input column
    int64_t o = (((int64_t)img * g.ho + wa0) * g.wo + wb) * c + ch;
    int64_t q = (((int64_t)img * g.h + 2 * wa0) * g.w + 2 * wb) * c + ch;
    // A row of two windows; one that does not exist has no winner.
    struct Windows { tsp::Raw8<T> dy[2]; uint2 tap[2]; };
    auto windows = [&](int64_t at, bool have, Windows& r) {
      r.tap[0] = r.tap[1] = make_uint2(0xffffffffu, 0xffffffffu);
      if (have) {
        tsp::ldraw(dy, at, r.dy[0]);
        r.tap[0] = *reinterpret_cast<const uint2*>(idx + at);
        if (right) {
          tsp::ldraw(dy, at + c, r.dy[1]);
          r.tap[1] = *reinterpret_cast<const uint2*>(idx + at + c);
        }
      }
    };
    auto pixels = [&](int64_t at, bool second, tsp::Raw8<T> (&r)[4]) {
      tsp::ldraw(x, at, r[0]);
      if (col1) tsp::ldraw(x, at + c, r[1]);
      if (second) {
        tsp::ldraw(x, at + in_pitch, r[2]);
        if (col1) tsp::ldraw(x, at + in_pitch + c, r[3]);
      }
    };
    Windows up = {}, down = {};
    tsp::Raw8<T> xr[4] = {};
    windows(o, true, up);
    pixels(q, 2 * wa0 + 1 < g.h, xr);
    windows(o + out_pitch, wa0 + 1 < g.ho, down);
#pragma unroll 1
    for (int wa = wa0; wa < end; ++wa) {
      // the next block of pixels and its lower windows are on their way while this block is computed
      const bool more = wa + 1 < end;
      Windows next = {};
      tsp::Raw8<T> nx[4] = {};
      if (more) {
        pixels(q + 2 * in_pitch, 2 * wa + 3 < g.h, nx);
        windows(o + 2 * out_pitch, wa + 2 < g.ho, next);
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {                                     // channels 2j and 2j + 1
        V gv[4];
        uint32_t code[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const Windows& row = k < 2 ? up : down;
          gv[k] = D::get(row.dy[k & 1], j);
          code[k] = __byte_perm(j < 2 ? row.tap[k & 1].x : row.tap[k & 1].y, 0, (j & 1) ? 0x3424 : 0x1404);
        }
        // what window (wa + kw / 2, wb + kw % 2) gives pixel (2 wa + k / 2, 2 wb + k % 2)
        auto part = [&](int k, int kw) {
          const int ky = (k >> 1) + 1 - 2 * (kw >> 1), kx = (k & 1) + 1 - 2 * (kw & 1);
          return D::keep(D::same_code(code[kw], tap_code(ky, kx)), gv[kw]);
        };
        V d[4];                                                         // rounded as a tensor of the sums would be
        d[0] = part(0, 0);
        d[1] = D::sum(part(1, 0), part(1, 1));
        d[2] = D::sum(part(2, 0), part(2, 2));
        d[3] = D::round((D::wide(part(3, 0)) + D::wide(part(3, 1))) + (D::wide(part(3, 2)) + D::wide(part(3, 3))));
#pragma unroll
        for (int k = 0; k < 4; ++k)
          D::set(xr[k], j, D::round(tsp::fma2(A[j], D::wide(d[k]), tsp::fma2(B[j], D::wide(D::get(xr[k], j)), C[j]))));
      }
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (((k & 1) == 0 || col1) && (k < 2 || 2 * wa + 1 < g.h)) st_raw(dx, q + (k >> 1) * in_pitch + (k & 1) * c, xr[k]);
      up = down;
      down = next;
#pragma unroll
      for (int k = 0; k < 4; ++k) xr[k] = nx[k];
      o += out_pitch;
      q += 2 * in_pitch;
    }
  }
}

// ---------------------------------------------------------------------------------------------
// Accumulated statistics of a partition's BatchNorm layers into the running ones (`batchnorm.py: BatchNormGroup`).  The views of
// a forward are taken one after the other: view g > 0 is added to set 0 first, and bit g of `commits` says whether the running
// statistics take what set 0 holds then, and set 0 starts over.  acc is [sum | sum of squares | count][set][channel].  Channels
// without a count keep their statistics.  A few kilobytes a layer, bound by launches: for the 53 layers of a ResNet-50, B200,
// 18 library kernels, 75 us with the gaps between them, and 2.5 us this way.
// ---------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(kBlock) bn_commit_kernel(float* __restrict__ acc, int sets, int total, int segs,
                                                           unsigned commits, const float* __restrict__ momentum,
                                                           float* __restrict__ mean_out, float* __restrict__ var_out,
                                                           long long* __restrict__ batches, int layers) {
  tsp::let_next_start();
  const int i = blockIdx.x * kBlock + threadIdx.x;
  if (i < layers) batches[i] += __popc(commits);
  if (i >= total) return;
  const int64_t per = (int64_t)sets * total;
  float v[3] = {acc[i], acc[per + i], acc[2 * per + i]}, rm = mean_out[i], rv = var_out[i];
  const float mom = momentum[i];
  for (int g = 0; g < segs; ++g) {
    if (g > 0) {
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        float* more = acc + q * per + (int64_t)g * total + i;
        v[q] += *more;
        *more = 0.f;
      }
    }
    if ((commits >> g & 1u) != 0) {
      if (v[2] > 0.f) {
        const float cnt = fmaxf(v[2], 1.f), mean = __fdiv_rn(v[0], cnt);
        const float var = __fsub_rn(__fdiv_rn(v[1], cnt), __fmul_rn(mean, mean));
        rm = __fadd_rn(rm, __fmul_rn(mean - rm, mom));
        rv = __fadd_rn(rv, __fmul_rn(var - rv, mom));
      }
      v[0] = v[1] = v[2] = 0.f;
    }
  }
#pragma unroll
  for (int q = 0; q < 3; ++q) acc[q * per + i] = v[q];
  if (commits != 0) {
    mean_out[i] = rm;
    var_out[i] = rv;
  }
}

// Row blocks of bn_colsum_kernel: enough to fill the chip four times over all slabs and segments, but at least one trip of
// `rows` rows per thread.
inline int row_blocks(int64_t m, int ty_n, int rows, int slabs, int segs) {
  const int64_t most = (m + (int64_t)ty_n * rows - 1) / ((int64_t)ty_n * rows);
  int64_t g = (148 * 4) / (slabs * segs);
  if (g > most) g = most;
  return (int)(g < 1 ? 1 : g);
}

// Blocks of the apply passes for one of `segs` groups: two blocks per SM over all groups before a thread takes a second
// vector, at most eight.
inline int apply_blocks(int64_t nvec, int cpv, int per_thread, int segs) {
  return tsp::row_stride_blocks(nvec, cpv, kBlock, per_thread, 148 * 2 / segs, 148 * 8 / segs);
}

// Streaming kernel eligibility: bf16, c/8 a power of two in [8, 256], enough rows to give every CTA work.
inline bool stream_ok(int64_t m, int c, int dtype) {
  const int cpv = c / 8;
  return dtype == TSP_DTYPE_BF16 && cpv >= 8 && cpv <= kStreamConsumers && (cpv & (cpv - 1)) == 0 &&
         m * (int64_t)c * 2 >= (1 << 20);
}

template <int MODE>
int launch_stream(const void* x, const void* dy, const void* y, void* dres, const float* mean_rstd, const float* w,
                  const float* bias, int relu, int64_t m, int c, int segs, float* sums, cudaStream_t stream) {
  const int narr = MODE == 0 ? 1 : (y != nullptr ? 3 : 2);
  const int64_t row_bytes = (int64_t)c * 2;
  // bytes per array and stage: 32 KB for one streamed array, 16 KB for two or three (at most 192 KB of ring);
  // smaller for small tensors so that every CTA still gets a few chunks to overlap
  int chunk = narr == 1 ? 32768 : 16384;
  while (chunk > 8192 && m * row_bytes < (int64_t)148 * 4 * chunk) chunk >>= 1;
  if (chunk < row_bytes) chunk = (int)row_bytes;
  const int64_t rows_per_chunk = chunk / row_bytes;
  int64_t grid = 148 / segs;                     // CTAs per segment: one CTA per SM over all segments
  if (grid < 1) grid = 1;
  const int64_t want = (m + 2 * rows_per_chunk - 1) / (2 * rows_per_chunk);
  if (want < grid) grid = want < 1 ? 1 : want;
  const size_t smem = (size_t)kStreamStages * narr * chunk + 2 * kStreamStages * 8 + kStreamConsumers * 16 * 4;
  auto kern = bn_colsum_stream_kernel<MODE>;
  static bool attr_set[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  dev &= 63;
  if (!attr_set[dev]) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 224 * 1024);
    if (e != cudaSuccess) return (int)e;
    attr_set[dev] = true;
  }
  kern<<<dim3((unsigned)grid, (unsigned)segs), kStreamThreads, smem, stream>>>((const __nv_bfloat16*)x, (const __nv_bfloat16*)dy,
                                                    (const __nv_bfloat16*)y, (__nv_bfloat16*)dres, mean_rstd, w, bias,
                                                    relu, m, c, chunk, sums);
  return TSP_LAUNCH_CHECK();
}

}  // namespace

extern "C" {

// 0 while no bounded wait of the streaming statistics kernels has run out on the current device; the first
// failing role otherwise (1 producer, 2 consumer).  Synchronises the device.  `reset` != 0 clears it.
int tsp_bn_stream_status(int reset) {
  int v = 0;
  if (cudaMemcpyFromSymbol(&v, g_bn_status, sizeof(int)) != cudaSuccess) return -1;
  if (reset && v != 0) {
    const int zero = 0;
    cudaMemcpyToSymbol(g_bn_status, &zero, sizeof(int));
  }
  return v;
}

// sums [2*c] fp32 is zeroed here, then receives per-channel sum(x) and sum(x^2).
// All four entry points take the activation as `segs` consecutive groups of m / segs rows; every group is
// normalised with its own statistics (two augmented views stacked along the batch axis).  Per-group arrays are
// laid out group-major: sums [segs][2c], save_mean_rstd [segs][2c].
int tsp_bn_stats(const void* x, int64_t m, int c, int dtype, float* sums, int segs, cudaStream_t stream) {
  if (m <= 0) return 0;
  if (c % 8 != 0 || c > 8192 || segs < 1 || m % segs != 0) return -3;
  cudaError_t e = cudaMemsetAsync(sums, 0, sizeof(float) * 2 * (size_t)c * segs, stream);
  if (e != cudaSuccess) return (int)e;
  m /= segs;
  if (stream_ok(m, c, dtype))
    return launch_stream<0>(x, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, 0, m, c, segs, sums, stream);
  const int cpv = c / 8;
  const Tile tl = make_tile(cpv);
  const int slabs = (cpv + tl.tx_n - 1) / tl.tx_n;
  const dim3 grid(row_blocks(m, tl.ty_n, (dtype == TSP_DTYPE_BF16 ? ColsumRows<__nv_bfloat16, 0>::value : ColsumRows<float, 0>::value), slabs, segs), slabs, segs);
  if (dtype == TSP_DTYPE_BF16)
    bn_colsum_kernel<__nv_bfloat16, 0><<<grid, kBlock, 0, stream>>>((const __nv_bfloat16*)x, nullptr, nullptr, nullptr,
                                                                       nullptr, nullptr, nullptr, 0, m, c, sums);
  else
    bn_colsum_kernel<float, 0><<<grid, kBlock, 0, stream>>>((const float*)x, nullptr, nullptr, nullptr, nullptr, nullptr,
                                                               nullptr, 0, m, c, sums);
  return TSP_LAUNCH_CHECK();
}

// sums [c] fp32 = (or, with `add`, +=) column sums of x [m, c] (the gradient of a bias).
int tsp_col_sums(const void* x, int64_t m, int c, int dtype, float* sums, int add, cudaStream_t stream) {
  return tsp_col_sums_of(&x, 1, m, c, dtype, sums, add, stream);
}

// The same of n_src (at most three) matrices of m rows and c columns each, in one launch: sums [n_src][c].  The gradients of q, k and
// v, 12608 rows of 768 columns each, B200, from memory: 22.5 us as three launches, 18.0 as one.
int tsp_col_sums_of(const void* const* x, int n_src, int64_t m, int c, int dtype, float* sums, int add, cudaStream_t stream) {
  if (m <= 0) return 0;
  if (c % 8 != 0 || c > 8192 || n_src < 1 || n_src > 3) return -3;
  cudaError_t e = add ? cudaSuccess : cudaMemsetAsync(sums, 0, sizeof(float) * (size_t)c * n_src, stream);
  if (e != cudaSuccess) return (int)e;
  const Tile tl = make_tile(c / 8);
  const int slabs = (c / 8 + tl.tx_n - 1) / tl.tx_n;
  const dim3 grid(row_blocks(m, tl.ty_n, (dtype == TSP_DTYPE_BF16 ? ColsumRows<__nv_bfloat16, 2>::value : ColsumRows<float, 2>::value), slabs, n_src), slabs, n_src);
  const void *x1 = n_src > 1 ? x[1] : nullptr, *x2 = n_src > 2 ? x[2] : nullptr;
  auto run = [&](auto kern, auto* p0, auto* p1, auto* p2) {
    kern<<<grid, kBlock, 0, stream>>>(p0, p1, p2, nullptr, nullptr, nullptr, nullptr, 0, m, c, sums);
  };
  using B = __nv_bfloat16;
  if (dtype == TSP_DTYPE_BF16) run(bn_colsum_kernel<B, 2>, (const B*)x[0], (const B*)x1, (const B*)x2);
  else run(bn_colsum_kernel<float, 2>, (const float*)x[0], (const float*)x1, (const float*)x2);
  return TSP_LAUNCH_CHECK();
}

// The per-channel vectors that a kernel reads 16 bytes at a time.
static bool vectors_ok(const void* a, const void* b, const void* c, const void* d) {
  return ((((uintptr_t)a) | ((uintptr_t)b) | ((uintptr_t)c) | ((uintptr_t)d)) & 15) == 0;
}

// w, b, sums and fixed_mean_var: 16-byte aligned.
// acc_sum / acc_sumsq / acc_count (optional): accumulators of the deferred running statistics; group g adds into
// acc + g * acc_seg_stride, so that each group's mini-batch can be committed on its own.
int tsp_bn_apply(const void* x, const void* res, void* y, const float* sums, const float* fixed_mean_var,
                 const float* w, const float* b, float* save_mean_rstd, float* acc_sum, float* acc_sumsq,
                 float* acc_count, int64_t acc_seg_stride, int64_t m, int c, float eps, int relu, int dtype, int segs,
                 cudaStream_t stream) {
  if (m <= 0) return 0;
  if (c % 8 != 0 || c > 4096 || segs < 1 || m % segs != 0) return -3;
  if (!vectors_ok(w, b, sums, fixed_mean_var)) return -2;
  m /= segs;
  const bool once = m * segs * c * (dtype == TSP_DTYPE_BF16 ? 2 : 4) <= kStaysInL2;
#define TSP_BN_APPLY(T, RES, ONCE)                                                                                      \
  bn_apply_kernel<T, RES, ONCE><<<dim3(apply_blocks(m * (c / 8), c / 8, RES ? ApplyVecs<T>::fwd_res : ApplyVecs<T>::fwd, segs), \
                                 segs), kBlock, 0, stream>>>(                                                            \
      (const T*)x, (const T*)res, (T*)y, sums, fixed_mean_var, w, b, save_mean_rstd, acc_sum, acc_sumsq, acc_count,      \
      acc_seg_stride, m, c, eps, relu)
#define TSP_BN_APPLY_RES(T)                                                                                             \
  if (res) { if (once) TSP_BN_APPLY(T, true, true); else TSP_BN_APPLY(T, true, false); }                                \
  else { if (once) TSP_BN_APPLY(T, false, true); else TSP_BN_APPLY(T, false, false); }
  if (dtype == TSP_DTYPE_BF16) { TSP_BN_APPLY_RES(__nv_bfloat16) } else { TSP_BN_APPLY_RES(float) }
#undef TSP_BN_APPLY_RES
#undef TSP_BN_APPLY
  return TSP_LAUNCH_CHECK();
}

// sums [segs][2*c], zeroed by the caller, receives per group sum(dy') and sum(dy' * xhat) (db and dw are their sums over
// the groups).  `y` non-null applies the ReLU mask; `dres` non-null receives dy'.
int tsp_bn_bwd_reduce(const void* dy, const void* x, const void* y, void* dres, const float* mean_rstd, const float* w,
                      const float* bias, int relu, int64_t m, int c, int dtype, float* sums, int segs,
                      cudaStream_t stream) {
  if (m <= 0) return 0;
  if (c % 8 != 0 || c > 8192 || segs < 1 || m % segs != 0) return -3;
  if (!vectors_ok(w, bias, mean_rstd, nullptr)) return -2;
  m /= segs;
  if (stream_ok(m, c, dtype))
    return launch_stream<1>(x, dy, y, dres, mean_rstd, w, bias, relu, m, c, segs, sums, stream);
  const int cpv = c / 8;
  const Tile tl = make_tile(cpv);
  const int slabs = (cpv + tl.tx_n - 1) / tl.tx_n;
  const dim3 grid(row_blocks(m, tl.ty_n, (dtype == TSP_DTYPE_BF16 ? ColsumRows<__nv_bfloat16, 1>::value : ColsumRows<float, 1>::value), slabs, segs), slabs, segs);
  if (dtype == TSP_DTYPE_BF16)
    bn_colsum_kernel<__nv_bfloat16, 1><<<grid, kBlock, 0, stream>>>((const __nv_bfloat16*)x, (const __nv_bfloat16*)dy,
                                                                       (const __nv_bfloat16*)y, (__nv_bfloat16*)dres,
                                                                       mean_rstd, w, bias, relu, m, c, sums);
  else
    bn_colsum_kernel<float, 1><<<grid, kBlock, 0, stream>>>((const float*)x, (const float*)dy, (const float*)y,
                                                               (float*)dres, mean_rstd, w, bias, relu, m, c, sums);
  return TSP_LAUNCH_CHECK();
}

// gw / gb (optional, together): the gradients of the weight and the bias are added to them.
int tsp_bn_bwd_apply(const void* dy, const void* x, const void* y, const float* mean_rstd, const float* w,
                     const float* bias, int relu, const float* sums, void* dx, float* gw, float* gb, int64_t m, int c,
                     int dtype, int segs, cudaStream_t stream) {
  if (m <= 0) return 0;
  if (c % 8 != 0 || c > 4096 || segs < 1 || m % segs != 0) return -3;
  if (!vectors_ok(w, bias, mean_rstd, sums)) return -2;
  m /= segs;
  const int mask = y != nullptr ? 2 : (relu ? 1 : 0);
#define TSP_BN_BWD(T, MASK)                                                                                             \
  bn_bwd_apply_kernel<T, MASK>                                                                                          \
      <<<dim3(apply_blocks(m * (c / 8), c / 8, ApplyVecs<T>::bwd, segs), segs), kBlock, 0, stream>>>(                   \
          (const T*)dy, (const T*)x, (const T*)y, mean_rstd, w, bias, sums, (T*)dx, gw, gb, m, c)
#define TSP_BN_BWD_MASK(T)                                                                                              \
  do { if (mask == 2) TSP_BN_BWD(T, 2); else if (mask == 1) TSP_BN_BWD(T, 1); else TSP_BN_BWD(T, 0); } while (0)
  if (dtype == TSP_DTYPE_BF16) TSP_BN_BWD_MASK(__nv_bfloat16);
  else TSP_BN_BWD_MASK(float);
#undef TSP_BN_BWD_MASK
#undef TSP_BN_BWD
  return TSP_LAUNCH_CHECK();
}

// One partition forward of `segs` views into the accumulators and running statistics (see bn_commit_kernel).
int tsp_bn_commit(float* acc, int sets, int total, int segs, unsigned commits, const float* momentum, float* running_mean,
                  float* running_var, long long* batches, int layers, cudaStream_t stream) {
  if (total <= 0 || layers > total || segs < 1 || segs > sets || segs > 32) return -3;
  bn_commit_kernel<<<(total + kBlock - 1) / kBlock, kBlock, 0, stream>>>(acc, sets, total, segs, commits, momentum, running_mean,
                                                                         running_var, batches, layers);
  return TSP_LAUNCH_CHECK();
}

// Training-mode BatchNorm + ReLU + 3x3 / 2 / 1 max-pool of x [segs * n, h, w, c] (statistics per group of n images, from
// `sums` [segs][2c] = sum and sum of squares over a group's pixels) -> y [segs * n, ho, wo, c], ho = (h + 1) / 2.  For the
// backward (together, optional, same shape as y): idx receives the winning taps, won the winners' elements of x.  The other
// arguments as in tsp_bn_apply.
static int pool_geom(int n, int h, int w, int c, int segs, PoolGeom* g) {
  if (n <= 0 || h < 1 || w < 1 || c % 8 != 0 || c > 4096 || segs < 1) return -3;
  const int ho = (h + 1) / 2, wo = (w + 1) / 2;
  if ((int64_t)n * (h + 1) * (w + 1) >= 0x7fffffff || (int64_t)w * c >= 0x7fffffff) return -3;
  // strips of four rows where they give an SM four blocks, of fewer rows on smaller tensors
  int rows = 4, sms = 0;
  if (cudaError_t e = tsp::usable_sms(sms); e != cudaSuccess) return (int)e;
  const int64_t blocks = (int64_t)segs * n * ho * wo * (c / 8) / kBlock;
  while (rows > 1 && blocks / rows < sms * 4) rows /= 2;
  const int strips = (ho + rows - 1) / rows;
  *g = {n, h, w, c, ho, wo, rows, FastDiv(wo), FastDiv(strips), (uint32_t)((int64_t)n * strips * wo)};
  return 0;
}

// Blocks for all items of a segment, at most `waves` per SM over all segments, and its segments and channel slabs.
static dim3 pool_grid(const PoolGeom& g, int segs, int waves) {
  const int cpv = g.c / 8, per_block = kBlock / (cpv < kBlock ? cpv : kBlock), slabs = (cpv + kBlock - 1) / kBlock;
  int64_t blocks = ((int64_t)g.items + per_block - 1) / per_block;
  const int64_t most = 148 * waves / ((int64_t)segs * slabs);
  if (blocks > most) blocks = most;
  return dim3((unsigned)(blocks < 1 ? 1 : blocks), (unsigned)segs, (unsigned)slabs);
}

int tsp_bn_relu_pool_fwd(const void* x, void* y, uint8_t* idx, void* won, const float* sums, const float* w, const float* b,
                         float* save_mean_rstd, float* acc_sum, float* acc_sumsq, float* acc_count, int64_t acc_seg_stride,
                         int n, int h, int wd, int c, float eps, int dtype, int segs, cudaStream_t stream) {
  PoolGeom g;
  const int rc = pool_geom(n, h, wd, c, segs, &g);
  if (rc != 0) return rc;
  if (!vectors_ok(w, b, sums, nullptr)) return -2;
  if ((idx == nullptr) != (won == nullptr)) return -3;
  const dim3 grid = pool_grid(g, segs, 32);
  auto run = [&](auto kern, auto* px, auto* py, auto* pw) {
    kern<<<grid, kBlock, 0, stream>>>(px, py, idx, pw, sums, w, b, save_mean_rstd, acc_sum, acc_sumsq, acc_count,
                                      acc_seg_stride, g, eps);
  };
  using B = __nv_bfloat16;
  if (dtype == TSP_DTYPE_BF16)
    run(idx != nullptr ? bn_relu_pool_kernel<B, true> : bn_relu_pool_kernel<B, false>, (const B*)x, (B*)y, (B*)won);
  else
    run(idx != nullptr ? bn_relu_pool_kernel<float, true> : bn_relu_pool_kernel<float, false>, (const float*)x, (float*)y,
        (float*)won);
  return TSP_LAUNCH_CHECK();
}

// Its backward: dy [segs * n, ho, wo, c], idx, won and x as above -> dx; sums [segs][2c], zeroed by the
// caller, receives db and dw; gw / gb as in tsp_bn_bwd_apply.
int tsp_bn_relu_pool_bwd(const void* dy, const uint8_t* idx, const void* won, const void* x, const float* mean_rstd,
                         const float* w, const float* b, float* sums, void* dx, float* gw, float* gb, int n, int h, int wd,
                         int c, int dtype, int segs, cudaStream_t stream) {
  PoolGeom g;
  int rc = pool_geom(n, h, wd, c, segs, &g);
  if (rc != 0) return rc;
  if (!vectors_ok(w, mean_rstd, sums, nullptr)) return -2;
  // The gradient meets the winners only, one per window: the two sums are those of a BatchNorm + ReLU over them.
  rc = tsp_bn_bwd_reduce(dy, won, nullptr, nullptr, mean_rstd, w, b, 1, (int64_t)segs * n * g.ho * g.wo, c, dtype, sums, segs,
                         stream);
  if (rc != 0) return rc;
  const dim3 grid = pool_grid(g, segs, 32);
  if (dtype == TSP_DTYPE_BF16) {
    using B = __nv_bfloat16;
    bn_relu_pool_bwd_kernel<B><<<grid, kBlock, 0, stream>>>((const B*)dy, idx, (const B*)x, mean_rstd, w, sums, (B*)dx, gw, gb,
                                                            g);
  } else {
    bn_relu_pool_bwd_kernel<float><<<grid, kBlock, 0, stream>>>((const float*)dy, idx, (const float*)x, mean_rstd, w, sums,
                                                                (float*)dx, gw, gb, g);
  }
  return TSP_LAUNCH_CHECK();
}

}  // extern "C"

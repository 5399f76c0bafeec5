// ResNet stem convolution on the 5th-generation tensor cores: y = conv2d(x, w), 7 x 7, stride 2, padding 3,
// 3 -> 64 channels, channels-last bf16, with the per-channel sum / sum of squares of y (the statistics of the
// BatchNorm that follows) accumulated in the epilogue.
//
// Reference call site: the first layer of torchvision's ResNet used by `benchmarks/byol/models/resnet_base_network.py`
// and `benchmarks/soft_target/models/resnet.py` (library convolution there).  The library's kernel for this
// shape pads 3 input channels to 8 and runs at a few percent of the machine; as an implicit GEMM the layer is
// M = N*OH*OW output pixels, N = 64, K = 7*7*3 = 147 and is bound by writing y.
//
// No patch matrix is built.  Image rows lie in a ring in shared memory with 4 channels per pixel (the fourth zero), 8 bytes
// a pixel, so at stride 2 the patch rows of consecutive output pixels start 16 bytes apart: one row is, as it lies, an
// unswizzled operand whose 8 x 16-byte core matrices overlap.  K-major (forward): pixel m, taps 2c, 2c+1 at byte 16 (m + c);
// MN-major (weight gradient): the same bytes with the pixel as the contraction index.  What shared memory sees per output
// row is then two rows written once instead of 128 patches of 320 bytes, whose accesses were the bound.  128 images of 224 x 224, the
// kernel alone: forward 136 us with a patch matrix written by 256 threads, 72 this way (31 to write y); weight gradient 115 and 72; 8
// images of 96 x 96 7.9 and 9.1, 9.4 and 9.0: a CTA has four output rows there at least, and one with patches.
//
// A tile is four output rows (n, oh) .. (n, oh + 3) of one image, OW <= 112 pixels each, i.e. eight more image rows (a batch)
// through the ring; one persistent CTA per SM walks a contiguous range of tiles.  The issuing thread is the serial resource: a
// commit and a barrier's wait cost it as much as several products (with a tile per output row, 14 products each, the forward
// took 119 us, and 90 with two of the 14), hence tiles of four rows and products over two output rows where there are two.
// What is left is the issuing thread's time and the statistics together (76 us, 56 without both, in repeated calls).
//
// Forward: a tap row takes two products of 16: taps 0..3 from the ring, and taps 3..6 from a copy of
// the ring that lies one pixel (8 bytes) earlier.  Tap 3 is in both with half its weight: with taps 4..7 in the second product
// the eighth would meet a zero weight, and an infinite pixel outside the window would make a NaN of it.  Image row r of a pair of
// output rows is tap row r of the first and r - 2 of the second: where both exist, one product with N = 128 serves both, its B
// operand the weights of tap rows r - 2 and r, which lie 64 rows apart in shared memory.
//   warps 0-7   rows: global memory -> ring, eight rows at a time, one per warp;
//   warp  8     one thread issues 19 x tcgen05.mma (128 x 64 or 128 x 128, x 16) per pair of rows, two accumulators of four
//               rows in tensor memory;
//   warps 9-16  epilogue, four per pair of rows: tcgen05.ld -> bf16 -> swizzled staging -> TMA store (3-d map, rows >= OW
//               clipped), and column sums of the staged block for the BatchNorm statistics.
//
// Weight gradient (conv_stem_wgrad_kernel): dW[co][k] += sum over pixels dY[p][co] * patch[p][k].  Products take a pair of output
// rows: M = 16 image rows x 8 (2 pixels of 4 channels), N = 2 rows of dY x 64 channels, one product per pair of taps c and 16
// pixels; row r of M and row j of dY belong to tap row r - 2j, the combinations outside 0..6 are not read.  The four 128 x
// 128 accumulators fill tensor memory over all rows of a CTA; their sums leave through shared memory as one bulk addition.
// Every mbarrier wait is bounded; a wait that runs out sets *status and all roles leave their loops.
#include <cuda.h>

#include "common.cuh"
#include "tcgen05.cuh"
#include "tspipe_kernels.h"

extern int g_tsp_sm_reserve;          // defined in peer.cu

namespace {

constexpr int kCout = 64;
constexpr int kK = 147;                   // 7 x 7 x 3
constexpr int kKPad = 192;                // row length of the weight matrix in memory
constexpr int kRows = 32;                 // image rows in the ring, in batches of 8
constexpr int kBatches = kRows / 8;
constexpr int kPitch = 1872;              // bytes of a row: 3 + 224 + 7 pixels of 8 bytes (see conv_stem_wgrad_kernel)
constexpr int kSlack = 256;               // operand rows past an image row's end are read (and not used)
constexpr int kMirror = 5;                // weight gradient: rows that follow the ring's end again, so that no tile wraps
constexpr int kRingBytes = kRows * kPitch + kSlack;
constexpr int kMBlockBytes = 128 * 128;   // 128 pixels x 64 channels of dY
constexpr int kBBlockBytes = kCout * 128;
constexpr int kBBytes = 4 * kBBlockBytes; // weights: 14 x 16 of the contraction, in blocks of 64
constexpr int kStoreBufBytes = 32 * 128;
// Epilogue warps: one per output row of a tile and TMEM lane quarter where statistics are formed and a CTA has tiles enough to make
// up for its larger start (128 images of 224 x 224, B200: 76.8 us with eight, 69 with sixteen; 37 of 192 x 192 22.9 and 22.0, 16 of
// 160 x 160 14.4 and 14.8, 8 of 96 x 96 9.1 and 10.2; without statistics 57 and 61), half of them with two rows each elsewhere.
constexpr int kManyWarps = 16, kFewWarps = 8, kManyTiles = 5;
constexpr int kWeightWarps = 8;          // of them, those that lay out the weights
constexpr int kStagingBytes = 16 * kStoreBufBytes;
constexpr int kTileRows = 4;
constexpr int kAccs = 2;
constexpr int kLoaders = 8;               // warps that fill the ring
__host__ __device__ constexpr int threads_with(int epi_warps) { return (kLoaders + 1 + epi_warps) * 32; }
constexpr int kSmemBytes = kBBytes + kStagingBytes + 2 * kRingBytes + 1024 + 256;
constexpr int kWgThreads = (kLoaders + 2) * 32;
constexpr int kWgRows = kRows - 4 + 16;   // rows that a product may touch from the last tile start on
constexpr int kDyStages = 2;
constexpr int kDyBytes = kTileRows * kMBlockBytes;
constexpr int kWgSmemBytes = kDyStages * kDyBytes + kWgRows * kPitch + kSlack + 1024 + 256;
constexpr uint64_t kWaitNs = 2000000000ull;
// the sums leave through the memory of the dY tiles: as they go out, and before that the two rows' parts [147][68], a pitch with
// which neither rows nor columns meet in a bank
constexpr int kPartPitch = kCout + 4, kPartFloats = kK * kPartPitch, kPartAt = 9408;
static_assert(kPartAt >= kCout * kK && (kPartAt + 2 * kPartFloats) * 4 <= kDyStages * kDyBytes, "sums and parts in two tiles of dY");
static_assert(kCout * kKPad * 2 <= kStagingBytes, "the weights in the staging buffers");

using tc5::mbar_arrive;
using tc5::mbar_expect_tx;
using tc5::mbar_init;
using tc5::smem_u32;

__device__ __forceinline__ void tma_load_3d(void* smem_dst, const CUtensorMap* map, uint64_t* bar, int x, int y, int z) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(map), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z)
      : "memory");
}
__device__ __forceinline__ void tma_store_3d(const CUtensorMap* map, const void* smem_src, int x, int y, int z) {
  asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%2, %3, %4}], [%1];" ::"l"(map),
               "r"(smem_u32(smem_src)), "r"(x), "r"(y), "r"(z)
               : "memory");
  asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}
// Unswizzled operand of 8 x 16-byte core matrices, any 16-byte aligned start.  K-major: `lbo` bytes to the next 8 along K,
// `sbo` to the next 8 rows; MN-major: `lbo` to the next 8 along K, `sbo` to the next 8 along M or N.
__device__ __forceinline__ uint64_t desc_plain(uint32_t smem_addr, uint32_t lbo, uint32_t sbo) {
  return (uint64_t)((smem_addr >> 4) & 0x3FFF) | (uint64_t)(lbo >> 4) << 16 | (uint64_t)(sbo >> 4) << 32 | (uint64_t)1 << 46;
}

// Barrier over the loading warps that also ANDs a flag.
__device__ __forceinline__ bool loaders_and(bool ok) {
  uint32_t out;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.b32 q, %1, 0;\n\t"
      "bar.red.and.pred p, 1, %2, q;\n\t"
      "selp.b32 %0, 1, 0, p;\n\t}"
      : "=r"(out)
      : "r"((uint32_t)ok), "n"(kLoaders * 32)
      : "memory");
  return out != 0;
}

// The work of a CTA, tiles [t, t_end), as one run of consecutive tiles per image.  Tile i of a run needs image rows
// 2 * first + 8 i - 3 .. + 9, batches i and i + 1 of the run.
struct Runs {
  int t, t_end, per_image;
  int n, first, tiles, batches;             // image, first output row, tiles and batches of the present run
  __device__ __forceinline__ Runs(int begin, int end, int tiles_per_image)
      : t(begin), t_end(end), per_image(tiles_per_image), n(0), first(0), tiles(0), batches(0) {}
  __device__ __forceinline__ bool next() {
    if (t >= t_end) return false;
    n = t / per_image;
    first = (t - n * per_image) * kTileRows;
    tiles = min(t_end, (n + 1) * per_image) - t;
    batches = tiles + 1;
    t += tiles;
    return true;
  }
};

// Warp `warp` of the loaders: its row of every batch.  SHIFTED: also the copy one pixel earlier.  Rows outside the image are
// zeros; the bytes left and right of a row's pixels are zeros from the start (zero_margins).  A batch's pixels are requested when
// the batch before it has been stored, the first one's by the constructor, while the block sets itself up.
template <bool SHIFTED>
struct RowLoader {
  const __nv_bfloat16* x;
  int h, w, warp, lane, k;
  Runs run;
  bool more;
  uint32_t v[4][3];
  __device__ __forceinline__ RowLoader(const __nv_bfloat16* __restrict__ x_, int h_, int w_, int per_image, int t_begin, int t_end,
                                       int warp_, int lane_)
      : x(x_), h(h_), w(w_), warp(warp_), lane(lane_), k(0), run(t_begin, t_end, per_image) {
    more = run.next();
    fetch();
  }
  __device__ __forceinline__ void fetch() {                    // of batch k of the present run
    const int ih = 2 * run.first - 3 + 8 * k + warp;
    const bool inside = more && ih >= 0 && ih < h;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int j = lane + 32 * i;
      v[i][0] = v[i][1] = v[i][2] = 0u;
      if (inside && 2 * j < w) {
        const uint32_t* src = reinterpret_cast<const uint32_t*>(x + ((int64_t)run.n * h + ih) * w * 3) + 3 * j;
        v[i][0] = __ldg(src); v[i][1] = __ldg(src + 1); v[i][2] = __ldg(src + 2);
      }
    }
  }
  __device__ __forceinline__ void store_all(uint8_t* ring, uint8_t* shifted, uint64_t* full_bar, uint64_t* empty_bar, int* status) {
    for (uint32_t gb = 0; more; ++gb) {
      const uint32_t b = gb % kBatches, round = gb / kBatches;
      if (round > 0 && !tc5::mbar_wait_warp(empty_bar + b, (round - 1) & 1, status, 1, kWaitNs, lane)) return;
      const int slot = (int)b * 8 + warp;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int j = lane + 32 * i;
        if (2 * j >= w) continue;
        const uint2 p0 = make_uint2(v[i][0], v[i][1] & 0xffffu);
        const uint2 p1 = make_uint2(__byte_perm(v[i][1], v[i][2], 0x5432), v[i][2] >> 16);
        uint8_t* at = ring + slot * kPitch + 24 + 16 * j;
        *reinterpret_cast<uint2*>(at) = p0;
        *reinterpret_cast<uint2*>(at + 8) = p1;
        if constexpr (SHIFTED) {
          *reinterpret_cast<uint4*>(shifted + slot * kPitch + 16 + 16 * j) = make_uint4(p0.x, p0.y, p1.x, p1.y);
        } else if (slot < kMirror) {
          *reinterpret_cast<uint2*>(at + kRows * kPitch) = p0;
          *reinterpret_cast<uint2*>(at + kRows * kPitch + 8) = p1;
        }
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(full_bar + b);
      if (++k == run.batches) { more = run.next(); k = 0; }
      fetch();
    }
  }
};
// Zeros in the pixels of `rows` ring rows before the first one, at `first`, and from the last one up to (not with) `end`: what taps
// outside the image read, and in the weight gradient what meets the zeros of dY past a row's end.  (What products read beyond, or
// of rows that no batch has filled, goes to results that are not used.)
__device__ __forceinline__ void zero_margins(uint8_t* ring, int rows, int first, int w, int end, int tid, int threads) {
  const int right = end - first - w, per_row = first + right;
  for (int i = tid; i < rows * per_row; i += threads) {
    const int row = i / per_row, at = i - row * per_row;
    *reinterpret_cast<uint2*>(ring + row * kPitch + 8 * (at < first ? at : w + at)) = make_uint2(0u, 0u);
  }
}

template <int EPI>
__global__ void __launch_bounds__(threads_with(EPI), 1)
conv_stem_kernel(const __nv_bfloat16* __restrict__ wmat, const __grid_constant__ CUtensorMap tmap_y,
                 const __nv_bfloat16* __restrict__ x, int n_img, int h, int w, int oh_n, int ow_n, int imgs_per_seg,
                 float* __restrict__ sums, int* __restrict__ status) {
  constexpr int kThreads = threads_with(EPI), kRowsEach = 16 / EPI;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* b_tile = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint8_t* store_bufs = b_tile + kBBytes;
  uint8_t* ring = store_bufs + kStagingBytes;
  uint8_t* shifted = ring + kRingBytes;
  uint64_t* bars = (uint64_t*)(shifted + kRingBytes);
  uint64_t* full_bar = bars;                     // [kBatches]  rows -> MMA (one arrival per loading warp)
  uint64_t* empty_bar = bars + kBatches;         // [kBatches]  MMA -> rows
  uint64_t* tmem_full_bar = bars + 2 * kBatches;             // [kAccs]
  uint64_t* tmem_empty_bar = bars + 2 * kBatches + kAccs;    // [kAccs]  8 arrivals
  uint64_t* weight_bar = bars + 2 * kBatches + 2 * kAccs;    // the weights as they lie in memory are here
  uint64_t* ready_bar = weight_bar + 1;                      // epilogue -> MMA: the weights as the products take them (8 arrivals)
  uint32_t* tmem_slot = (uint32_t*)(ready_bar + 1);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int per_image = (oh_n + kTileRows - 1) / kTileRows, num_tiles = n_img * per_image;
  const int per_cta = (num_tiles + gridDim.x - 1) / gridDim.x;
  const int t_begin = blockIdx.x * per_cta;
  const int t_end = t_begin + per_cta < num_tiles ? t_begin + per_cta : num_tiles;

  if (tid == 0) {
    for (int b = 0; b < kBatches; ++b) { mbar_init(full_bar + b, kLoaders); mbar_init(empty_bar + b, 1); }
    for (int a = 0; a < kAccs; ++a) { mbar_init(tmem_full_bar + a, 1); mbar_init(tmem_empty_bar + a, EPI); }
    mbar_init(weight_bar, 1);
    mbar_init(ready_bar, kWeightWarps);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    mbar_expect_tx(weight_bar, kCout * kKPad * 2);
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(store_bufs)),
                 "l"(wmat), "r"((uint32_t)(kCout * kKPad * 2)), "r"(smem_u32(weight_bar))
                 : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&tmap_y) : "memory");
  }
  RowLoader<true> loader(x, h, w, per_image, t_begin, warp < kLoaders ? t_end : t_begin, warp, lane);
  zero_margins(ring, kRows, 3, w, w + 8, tid, kThreads);
  zero_margins(shifted, kRows, 2, w, w + 8, tid, kThreads);
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  if (warp == kLoaders) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"((uint32_t)(kAccs * kTileRows * kCout))
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = *tmem_slot;

  if (warp < kLoaders) {
    loader.store_all(ring, shifted, full_bar, empty_bar, status);
  } else if (warp == kLoaders) {
    // ---------------- MMA issuer ----------------
    {
      const bool issuer = tc5::elect_one();
      constexpr uint32_t idesc1 = tc5::make_idesc(128, kCout, false, false), idesc2 = tc5::make_idesc(128, 2 * kCout, false, false);
      const uint64_t a0 = desc_plain(smem_u32(ring), 16, 128), a1 = desc_plain(smem_u32(shifted) + 16, 16, 128);
      const uint64_t b0 = tc5::desc_k_major(smem_u32(b_tile));
      // weights of tap row kh, product `half` of the two; 64 rows further on (the second half of N = 128): tap row kh + 2
      auto weights = [&](int kh, int half) -> uint64_t {
        return b0 + (uint64_t)((kh >> 1) * (kBBlockBytes / 16) + 4 * (kh & 1) + 2 * half);
      };
      uint32_t it = 0, base = 0, have = 0;                     // tiles; batches before this run, waited for
      bool ok = __all_sync(0xffffffffu, tc5::mbar_wait(ready_bar, 0, status, 2, kWaitNs)) != 0;
      Runs run(t_begin, t_end, per_image);
      while (ok && run.next()) {
        for (int i = 0; i < run.tiles && ok; ++i, ++it) {
          const uint32_t batch = base + i;                     // the tile's rows: this batch and the next one
          for (; ok && have <= batch + 1; ++have)
            ok = __all_sync(0xffffffffu, tc5::mbar_wait(full_bar + have % kBatches, (have / kBatches) & 1, status, 2, kWaitNs));
          const uint32_t acc = it % kAccs, use = it / kAccs;
          if (ok && use > 0) ok = __all_sync(0xffffffffu, tc5::mbar_wait(tmem_empty_bar + acc, (use - 1) & 1, status, 4, kWaitNs));
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const int rows = oh_n - run.first - kTileRows * i;   // output rows left in the image
#pragma unroll 1
          for (int p = 0; issuer && p < 2 && 2 * p < rows; ++p) {
            // columns 0..63: the pair's second row, 64..127: its first
            const uint32_t d = tmem_base + (acc * 2 + p) * 2 * kCout;
#pragma unroll
            for (int r = 0; r < 9; ++r) {
              const uint64_t row = (uint64_t)((batch * 8 + 4 * p + r) % kRows * (kPitch / 16));
#pragma unroll
              for (int half = 0; half < 2; ++half) {
                const uint64_t a = (half == 0 ? a0 : a1) + row;
                if (r < 2 || (r == 2 && half == 0)) tc5::umma_bf16(d + kCout, a, weights(r, half), idesc1, r > 0 || half > 0 ? 1u : 0u);
                if (r == 2 && half == 0) tc5::umma_bf16(d, a, weights(0, 0), idesc1, 0u);
                if (r > 6) tc5::umma_bf16(d, a, weights(r - 2, half), idesc1, 1u);
                if ((r > 2 && r < 7) || (r == 2 && half == 1)) tc5::umma_bf16(d, a, weights(r - 2, half), idesc2, 1u);
              }
            }
          }
          if (issuer) {
            tc5::umma_commit(tmem_full_bar + acc);
            tc5::umma_commit(empty_bar + batch % kBatches);
            if (i + 1 == run.tiles) tc5::umma_commit(empty_bar + (batch + 1) % kBatches);
          }
          __syncwarp();
        }
        base += run.batches;
      }
    }
  } else {
    // ---------------- epilogue: warps from 9 on, TMEM lanes 32*(warp%4) .. +31; group g takes the g-th kRowsEach of a tile's rows ----------------
    // First the weights as the products take them, while the loaders fill the ring: step 2 kh + half, element 4 * tap + channel, taps
    // 0..3 and 3..6 (128-byte swizzle), from a copy in the staging buffers.  (By all warps before their roles began, from
    // memory element by element, they made every call 2 us longer: 8 images of 96 x 96 10.8 us, 9.1 this way.)
    const __nv_bfloat16* raw = reinterpret_cast<const __nv_bfloat16*>(store_bufs);
    if (warp <= kLoaders + kWeightWarps) {
      tc5::mbar_wait(weight_bar, 0, status, 6, kWaitNs);
      const int e = tid - (kLoaders + 1) * 32, kh = (e >> 3) & 7, half = (e >> 2) & 1, tap = 3 * half + (e & 3);
      const int step = 2 * kh + half, piece = 2 * (step & 3) + ((e >> 1) & 1);
      const __nv_bfloat16* at = raw + kh * 21 + tap * 3;
      uint8_t* to = b_tile + (step >> 2) * kBBlockBytes + 8 * (e & 1);
#pragma unroll 1
      for (int co0 = e >> 6; kh < 7 && co0 < kCout; co0 += 32) {         // this tap of eight rows, all loads before the first store
        __nv_bfloat162 v[8][2];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const __nv_bfloat16* src = at + (co0 + 4 * k) * kKPad;
          v[k][0] = __halves2bfloat162(src[0], src[1]);
          v[k][1] = __halves2bfloat162(src[2], __float2bfloat16(0.f));
        }
        if (tap == 3) {        // the two halves add up to the weight: both the same but for the last bit of a subnormal
#pragma unroll
          for (int k = 0; k < 16; ++k) {
            __nv_bfloat162& x = v[k >> 1][k & 1];
            const __nv_bfloat162 one = __hmul2(x, __float2bfloat162_rn(0.5f)), other = __hsub2(x, one);
            x = half == 0 ? one : __halves2bfloat162(__hisinf(one.x) ? one.x : other.x, __hisinf(one.y) ? one.y : other.y);
          }
        }
#pragma unroll
        for (int k = 0; k < 8; ++k)
          *reinterpret_cast<uint2*>(to + (co0 + 4 * k) * 128 + ((piece ^ ((co0 + 4 * k) & 7)) << 4)) =
              make_uint2(*reinterpret_cast<const uint32_t*>(&v[k][0]), *reinterpret_cast<const uint32_t*>(&v[k][1]));
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(ready_bar);
    }
    const int quarter = warp & 3, group = (warp - kLoaders - 1) >> 2;
    uint8_t* bufs = store_bufs + (warp - kLoaders - 1) * kRowsEach * kStoreBufBytes;      // a staging block per row
    tc5::ColSums cs;
    cs.clear();
    int cur_seg = -1;
    auto flush_sums = [&]() {
      if (sums != nullptr && cur_seg >= 0) {
        float v[2], q[2];
        cs.reduce(lane, v, q);
        float* dst = sums + cur_seg * 2 * kCout + tc5::ColSums::channel(lane);
        atomicAdd(dst, v[0]);
        atomicAdd(dst + 1, v[1]);
        atomicAdd(dst + kCout, q[0]);
        atomicAdd(dst + kCout + 1, q[1]);
      }
      cs.clear();
    };
    const int row0 = quarter * 32;
    uint32_t stores = 0;
    bool ok = true;
    for (int t = t_begin; t < t_end && ok; ++t) {
      const uint32_t it = t - t_begin, first_store = stores;
      const int n = t / per_image, oh = (t - n * per_image) * kTileRows + kRowsEach * group;
      const int seg = n / imgs_per_seg;                    // statistics are kept per group of images
      if (seg != cur_seg) { flush_sums(); cur_seg = seg; }
      const uint32_t acc = it % kAccs;
      ok = tc5::mbar_wait_warp(tmem_full_bar + acc, (it / kAccs) & 1, status, 3, kWaitNs, lane);   // one way out per warp
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll 1
      for (int j = 0; j < kRowsEach && oh + j < oh_n; ++j) {
        const int row = kRowsEach * group + j;             // of the tile: columns 64..127 of its pair's accumulator are the first one's
        const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + (acc * 2 + (row >> 1)) * 2 * kCout + ((row & 1) == 0 ? kCout : 0);
        uint8_t* buf = bufs + stores++ % kRowsEach * kStoreBufBytes;
        if (lane == 0) {                                   // the last store from it has read it
          if (kRowsEach == 1) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
          else asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
        }
        __syncwarp();
        uint8_t* my_row = buf + lane * 128;
        const bool keep = row0 + lane < ow_n;              // (the products' rows past the output row hold what lies there)
#pragma unroll
        for (int hc = 0; hc < 2; ++hc) {                   // 32 channels (the sums of 8 channels take 32 registers as it is)
          uint32_t r[32];
          tc5::tmem_ld_32x32_issue(taddr + 32 * hc, r);
          tc5::tmem_ld_wait();
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            uint4 v = make_uint4(0u, 0u, 0u, 0u);
            if (keep) {
              v.x = tc5::pack_bf16x2(__uint_as_float(r[8 * q + 0]), __uint_as_float(r[8 * q + 1]));
              v.y = tc5::pack_bf16x2(__uint_as_float(r[8 * q + 2]), __uint_as_float(r[8 * q + 3]));
              v.z = tc5::pack_bf16x2(__uint_as_float(r[8 * q + 4]), __uint_as_float(r[8 * q + 5]));
              v.w = tc5::pack_bf16x2(__uint_as_float(r[8 * q + 6]), __uint_as_float(r[8 * q + 7]));
            }
            *reinterpret_cast<uint4*>(my_row + (((4 * hc + q) ^ (lane & 7)) << 4)) = v;
          }
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0) {
          if (row0 < ow_n) tma_store_3d(&tmap_y, buf, 0, row0, n * oh_n + oh + j);
          else asm volatile("cp.async.bulk.commit_group;" ::: "memory");
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(tmem_empty_bar + acc);
      if (sums != nullptr)                                 // statistics of the rounded outputs, the accumulator being free again
        for (int j = 0; j < kRowsEach && oh + j < oh_n; ++j) cs.add(bufs + (first_store + j) % kRowsEach * kStoreBufBytes, lane);
    }
    if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    __syncwarp();
    // the last sums go through the staging buffer and leave as one addition per channel and CTA (below)
    float* st = reinterpret_cast<float*>(bufs);
    float v[2], q[2];
    cs.reduce(lane, v, q);
    *reinterpret_cast<float2*>(st + tc5::ColSums::channel(lane)) = make_float2(v[0], v[1]);
    *reinterpret_cast<float2*>(st + kCout + tc5::ColSums::channel(lane)) = make_float2(q[0], q[1]);
    if (lane == 0) st[2 * kCout] = __int_as_float(ok ? cur_seg : -1);
  }
  if (*((volatile int*)status) != 0) tc5::drain_in_flight();
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (sums != nullptr && tid < 2 * kCout) {
    // (additions to one sector are serialised: 8 warps x 2 instructions from each of 148 CTAs cost some 30 us)
    const float* st = reinterpret_cast<const float*>(store_bufs);
    constexpr int kWarpFloats = kRowsEach * kStoreBufBytes / 4;
    const int seg = __float_as_int(st[2 * kCout]);
    bool same = seg >= 0;
    float v = 0.f;
    for (int q = 0; q < EPI; ++q) {
      v += st[q * kWarpFloats + tid];
      same = same && __float_as_int(st[q * kWarpFloats + 2 * kCout]) == seg;      // (else a wait ran out)
    }
    if (same) atomicAdd(sums + seg * 2 * kCout + tid, v);
  }
  if (warp == kLoaders) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)(kAccs * kTileRows * kCout)) : "memory");
  }
}

// The share of tiles [t_begin, t_end) in the sums of tap row kh from the definition (a tap's pixels outside the image are zeros),
// by a warp, for those of `sum` [co][147] that are not finite: lane = two output channels, all 21 taps and input channels of the row
// in registers, so that dY is read once per tap row, 128 bytes at a time (128 images of 218 x 216: 5 ms, once there is one).
__device__ __noinline__ void exact_tap_row(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ dy, int h, int w,
                                           int oh_n, int ow_n, int per_image, int t_begin, int t_end, int kh, int lane, float* sum) {
  constexpr int kTaps = 21;
  float acc[kTaps][2];
#pragma unroll
  for (int k = 0; k < kTaps; ++k) acc[k][0] = acc[k][1] = 0.f;
  for (int t = t_begin; t < t_end; ++t) {
    const int n = t / per_image, oh0 = (t - n * per_image) * kTileRows;
    for (int oh = oh0; oh < oh0 + kTileRows && oh < oh_n; ++oh) {
      const int ih = 2 * oh - 3 + kh;
      const bool inside = ih >= 0 && ih < h;
      const __nv_bfloat16* xr = x + ((int64_t)n * h + (inside ? ih : 0)) * w * 3;
      const uint32_t* dr = reinterpret_cast<const uint32_t*>(dy + ((int64_t)n * oh_n + oh) * ow_n * kCout) + lane;
      float part[kTaps][2];                    // of an output row
#pragma unroll
      for (int k = 0; k < kTaps; ++k) part[k][0] = part[k][1] = 0.f;
#pragma unroll 2
      for (int ox = 0; ox < ow_n; ++ox) {
        const int at = (2 * ox - 3) * 3 + lane;              // lane = (tap, channel) of the row
        const float mine = inside && lane < kTaps && at >= 0 && at < 3 * w ? __bfloat162float(xr[at]) : 0.f;
        const uint32_t d = __ldg(dr + ox * (kCout / 2));
        const float d0 = __uint_as_float(d << 16), d1 = __uint_as_float(d & 0xffff0000u);
#pragma unroll
        for (int k = 0; k < kTaps; ++k) {
          const float v = __shfl_sync(0xffffffffu, mine, k);
          part[k][0] = fmaf(d0, v, part[k][0]);
          part[k][1] = fmaf(d1, v, part[k][1]);
        }
      }
#pragma unroll
      for (int k = 0; k < kTaps; ++k) { acc[k][0] += part[k][0]; acc[k][1] += part[k][1]; }
    }
  }
#pragma unroll
  for (int k = 0; k < kTaps; ++k)
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      float* at = sum + (2 * lane + e) * kK + kh * kTaps + k;
      if ((__float_as_uint(*at) & 0x7f800000u) == 0x7f800000u) *at = acc[k][e];
    }
}

// The pitch of a row is an odd multiple of 16 bytes: what a product reads of one pixel, 16 bytes of each of 16 rows, then lies in
// all banks (with a pitch of 29 x 64 bytes in two 16-byte columns of them: 103 us, 97 this way, 82 issued by an elected lane).
// dw[co][147] (fp32) += sum over this CTA's output rows of dY^T patch.  Accumulator c (columns 128 c ..): lane 8 r + 4 dx + ch,
// column 64 j + co holds tap row r - 2 j, tap 2 c + dx.
__global__ void __launch_bounds__(kWgThreads, 1)
conv_stem_wgrad_kernel(const __grid_constant__ CUtensorMap tmap_dy, const __nv_bfloat16* __restrict__ x,
                       const __nv_bfloat16* __restrict__ dy, int n_img, int h, int w, int oh_n, int ow_n, float* __restrict__ dw, int* __restrict__ status) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* dy_tiles = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint8_t* ring = dy_tiles + kDyStages * kDyBytes;
  uint64_t* bars = (uint64_t*)(ring + kWgRows * kPitch + kSlack);
  uint64_t* full_bar = bars;                         // [kBatches]   rows -> MMA
  uint64_t* empty_bar = bars + kBatches;             // [kBatches]   MMA -> rows
  uint64_t* dy_full_bar = bars + 2 * kBatches;               // [kDyStages]  dY loads -> MMA
  uint64_t* dy_empty_bar = bars + 2 * kBatches + kDyStages;  // [kDyStages]  MMA -> dY loads
  uint64_t* done_bar = bars + 2 * kBatches + 2 * kDyStages;  // every product has completed
  uint32_t* tmem_slot = (uint32_t*)(done_bar + 1);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int per_image = (oh_n + kTileRows - 1) / kTileRows, num_tiles = n_img * per_image;
  const int per_cta = (num_tiles + gridDim.x - 1) / gridDim.x;
  const int t_begin = blockIdx.x * per_cta;
  const int t_end = t_begin + per_cta < num_tiles ? t_begin + per_cta : num_tiles;

  if (tid == 0) {
    for (int b = 0; b < kBatches; ++b) { mbar_init(full_bar + b, kLoaders); mbar_init(empty_bar + b, 1); }
    for (int s = 0; s < kDyStages; ++s) { mbar_init(dy_full_bar + s, 1); mbar_init(dy_empty_bar + s, 1); }
    mbar_init(done_bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&tmap_dy) : "memory");
  }
  RowLoader<false> loader(x, h, w, per_image, t_begin, warp < kLoaders ? t_end : t_begin, warp, lane);
  zero_margins(ring, kWgRows, 3, w, 2 * ((ow_n + 15) & ~15) + 8, tid, kWgThreads);
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  if (warp == kLoaders) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(512u)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = *tmem_slot;

  if (warp < kLoaders) {
    loader.store_all(ring, nullptr, full_bar, empty_bar, status);
    // ---------------- epilogue: TMEM lanes 32 * (warp % 4) .. + 31; the first four warps take the pair's first row, the others its second ----------------
    // (after a wait that ran out the accumulators hold part of their sums, or nothing: none of it is added)
    if (t_begin < t_end) {
      float* sum = reinterpret_cast<float*>(dy_tiles);         // [co][147]; every tile of dY has been used
      float* parts = sum + kPartAt;
      const bool good = tc5::mbar_wait_warp(done_bar, 0, status, 3, kWaitNs, lane) && *((volatile int*)status) == 0;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      // (Through a [co][147] matrix into which the second row's part was added, element by element, this took 12 us: 128 images 84.3 us,
      // 72 this way, 8 images of 96 x 96 21.4 and 9.0.)
      const int m = (warp & 3) * 32 + lane, dx = (m >> 2) & 1, ch = m & 3, j = warp >> 2;
      const int kh = (m >> 3) - 2 * j;
#pragma unroll 1
      for (int c = 0; c < 4; ++c) {
        uint32_t r[64];
        const uint32_t taddr = tmem_base + ((uint32_t)((warp & 3) * 32) << 16) + c * 128 + j * kCout;
        tc5::tmem_ld_32x32_issue(taddr, r);
        tc5::tmem_ld_32x32_issue(taddr + 32, r + 32);
        tc5::tmem_ld_wait();
        const int kw = 2 * c + dx;
        if (kh >= 0 && kh < 7 && kw < 7 && ch < 3) {
          float4* dst = reinterpret_cast<float4*>(parts + j * kPartFloats + (kh * 21 + kw * 3 + ch) * kPartPitch);
#pragma unroll
          for (int q = 0; q < kCout / 4; ++q)
            dst[q] = make_float4(__uint_as_float(r[4 * q]), __uint_as_float(r[4 * q + 1]), __uint_as_float(r[4 * q + 2]),
                                 __uint_as_float(r[4 * q + 3]));
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      if (loaders_and(good)) {
        bool finite = true;
#pragma unroll 5
        for (int i = warp; i < 2 * kK; i += kLoaders) {            // lane = output channel, of the first half or the second
          const int k = i >> 1, co = 32 * (i & 1) + lane;
          const float v = parts[k * kPartPitch + co] + parts[k * kPartPitch + co + kPartFloats];
          sum[co * kK + k] = v;
          finite = finite && (__float_as_uint(v) & 0x7f800000u) != 0x7f800000u;
        }
        // Zeros of dY past a row's end and of a missing row meet pixels too: an infinite or NaN one makes a NaN (0 x inf) of taps
        // that do not pair it with a dY.  Where there are such zeros, sums that are not finite are formed again.
        if (((ow_n & 15) != 0 || (oh_n & 1) != 0) && !loaders_and(finite) && warp < 7)
          exact_tap_row(x, dy, h, w, oh_n, ow_n, per_image, t_begin, t_end, warp, lane, sum);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        loaders_and(true);
        if ((reinterpret_cast<uintptr_t>(dw) & 15) == 0) {
          if (tid == 0) {
            asm volatile("cp.reduce.async.bulk.global.shared::cta.bulk_group.add.f32 [%0], [%1], %2;" ::"l"(dw),
                         "r"(smem_u32(sum)), "r"((uint32_t)(kCout * kK * 4))
                         : "memory");
            asm volatile("cp.async.bulk.commit_group;" ::: "memory");
            asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
          }
        } else {
          for (int i = tid; i < kCout * kK; i += kLoaders * 32) atomicAdd(dw + i, sum[i]);
        }
      }
    }
  } else if (warp == kLoaders) {
    // ---------------- MMA issuer ----------------
    {
      const bool issuer = tc5::elect_one();
      constexpr uint32_t idesc = tc5::make_idesc(128, 128, true, true);
      const int ksteps = (ow_n + 15) >> 4;                     // (dY is zero past the row's end, as are the ring's bytes there)
      const uint64_t a0 = desc_plain(smem_u32(ring), 128, kPitch);
      const uint64_t d0 = tc5::desc_mn_major(smem_u32(dy_tiles), kMBlockBytes);
      uint32_t it = 0, base = 0, have = 0;
      bool ok = true;
      Runs run(t_begin, t_end, per_image);
      while (ok && run.next()) {
        for (int i = 0; i < run.tiles && ok; ++i, ++it) {
          const uint32_t batch = base + i;
          for (; ok && have <= batch + 1; ++have)
            ok = __all_sync(0xffffffffu, tc5::mbar_wait(full_bar + have % kBatches, (have / kBatches) & 1, status, 2, kWaitNs));
          const uint32_t s = it % kDyStages;
          ok = ok && __all_sync(0xffffffffu, tc5::mbar_wait(dy_full_bar + s, (it / kDyStages) & 1, status, 4, kWaitNs));
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const int rows = oh_n - run.first - kTileRows * i;
#pragma unroll 1
          for (int p = 0; issuer && p < 2 && 2 * p < rows; ++p) {        // a pair's rows: 8 batch + 4 p .. + 8
            const uint64_t a = a0 + (uint64_t)((batch * 8 + 4 * p) % kRows * (kPitch / 16));
            const uint64_t d = d0 + (uint64_t)(s * (kDyBytes / 16) + p * (2 * kMBlockBytes / 16));
            for (int ks = 0; ks < ksteps; ++ks) {              // 16 pixels further on: +256 bytes of the ring, +2048 of dY
#pragma unroll
              for (int c = 0; c < 4; ++c)
                tc5::umma_bf16(tmem_base + c * 128, a + (uint64_t)(16 * ks + c), d + (uint64_t)(128 * ks), idesc,
                               it > 0 || p > 0 || ks > 0 ? 1u : 0u);
            }
          }
          if (issuer) {
            tc5::umma_commit(dy_empty_bar + s);
            tc5::umma_commit(empty_bar + batch % kBatches);
            if (i + 1 == run.tiles) tc5::umma_commit(empty_bar + (batch + 1) % kBatches);
          }
          __syncwarp();
        }
        base += run.batches;
      }
      if (issuer) tc5::umma_commit(done_bar);
    }
  } else {
    // ---------------- dY rows by TMA (missing ones: zeros, from past the tensor's end) ----------------
    if (lane == 0) {
      uint32_t it = 0;
      for (int t = t_begin; t < t_end; ++t, ++it) {
        const int s = it % kDyStages;
        const uint32_t round = it / kDyStages;
        if (round > 0 && !tc5::mbar_wait_parked(dy_empty_bar + s, (round - 1) & 1, status, 5, kWaitNs)) break;
        mbar_expect_tx(dy_full_bar + s, (uint32_t)kDyBytes);
        const int n = t / per_image, oh = kTileRows * (t - n * per_image);
        for (int j = 0; j < kTileRows; ++j)
          tma_load_3d(dy_tiles + s * kDyBytes + j * kMBlockBytes, &tmap_dy, dy_full_bar + s, 0, 0,
                      oh + j < oh_n ? n * oh_n + oh + j : n_img * oh_n);
      }
    }
  }
  if (*((volatile int*)status) != 0) tc5::drain_in_flight();
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == kLoaders) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
  }
}

}  // namespace

extern "C" {

// y[n, oh, ow, 64] = conv7x7/2 pad 3 of x[n, h, w, 3] (both bf16, channels-last memory) with wmat[64][192] bf16:
// wmat[oc][kh*21 + kw*3 + c] = weight[oc][c][kh][kw], zero beyond k = 146.  h even, w % 8 == 0, 8 <= w <= 224.
// `sums` (optional, [segs][128] floats, zeroed by the caller) receives per-channel sum and sum of squares of y for
// each of the `segs` consecutive groups of n / segs images.
// `status`: one zeroed int in device memory; non-zero afterwards = a bounded wait ran out and y is not valid.
int tsp_conv_stem_fwd(const void* x, const void* wmat, void* y, float* sums, int n, int h, int w, int segs,
                      int* status, cudaStream_t stream) {
  if (n <= 0) return 0;
  if (segs < 1 || n % segs != 0) return -3;
  if ((h & 1) || (w & 7) || w > 224 || h < 8 || w < 8) return -3;
  if ((((uintptr_t)x | (uintptr_t)wmat | (uintptr_t)y) & 15) != 0) return -2;
  const int oh = h / 2, ow = w / 2;
  CUtensorMap ty;
  {
    const cuuint64_t dims[3] = {(cuuint64_t)kCout, (cuuint64_t)ow, (cuuint64_t)n * oh};
    const cuuint64_t strides[2] = {(cuuint64_t)kCout * 2, (cuuint64_t)ow * kCout * 2};
    const cuuint32_t box[3] = {(cuuint32_t)kCout, 32, 1};
    if (!tc5::encode_tiled(&ty, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, y, 3, dims, strides, box, CU_TENSOR_MAP_L2_PROMOTION_NONE))
      return -6;
  }
  static bool attr_set[64] = {};
  static int n_sm[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  dev &= 63;
  if (!attr_set[dev]) {
    cudaError_t e = cudaFuncSetAttribute(conv_stem_kernel<kFewWarps>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(conv_stem_kernel<kManyWarps>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes);
    if (e != cudaSuccess) return (int)e;
    cudaDeviceGetAttribute(&n_sm[dev], cudaDevAttrMultiProcessorCount, dev);
    if (n_sm[dev] <= 0) n_sm[dev] = 148;
    attr_set[dev] = true;
  }
  const int tiles = n * ((oh + kTileRows - 1) / kTileRows);
  const int usable = n_sm[dev] - g_tsp_sm_reserve > 8 ? n_sm[dev] - g_tsp_sm_reserve : 8;
  const int grid = tiles < usable ? tiles : usable;
  auto run = [&](auto kern, int threads) {
    kern<<<grid, threads, kSmemBytes, stream>>>((const __nv_bfloat16*)wmat, ty, (const __nv_bfloat16*)x, n, h, w, oh, ow, n / segs,
                                                sums, status);
  };
  if (sums != nullptr && tiles >= kManyTiles * usable) run(conv_stem_kernel<kManyWarps>, threads_with(kManyWarps));
  else run(conv_stem_kernel<kFewWarps>, threads_with(kFewWarps));
  return TSP_LAUNCH_CHECK();
}

// dw[64][7][7][3] (fp32) += the weight gradient of tsp_conv_stem_fwd given its input x and dy [n, h/2, w/2, 64] (bf16,
// channels-last).
int tsp_conv_stem_wgrad(const void* x, const void* dy, float* dw, int n, int h, int w, int* status, cudaStream_t stream) {
  if (n <= 0) return 0;
  if ((h & 1) || (w & 7) || w > 224 || h < 8 || w < 8) return -3;
  if ((((uintptr_t)x | (uintptr_t)dy) & 15) != 0) return -2;
  const int oh = h / 2, ow = w / 2;
  CUtensorMap td;
  {
    cuuint64_t dims[3] = {(cuuint64_t)kCout, (cuuint64_t)ow, (cuuint64_t)n * oh};
    cuuint64_t strides[2] = {(cuuint64_t)kCout * 2, (cuuint64_t)ow * kCout * 2};
    cuuint32_t box[3] = {(cuuint32_t)kCout, 128, 1};
    if (!tc5::encode_tiled(&td, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, dy, 3, dims, strides, box, CU_TENSOR_MAP_L2_PROMOTION_L2_256B))
      return -6;
  }
  static bool attr_set[64] = {};
  static int n_sm[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  dev &= 63;
  if (!attr_set[dev]) {
    cudaError_t e = cudaFuncSetAttribute(conv_stem_wgrad_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kWgSmemBytes);
    if (e != cudaSuccess) return (int)e;
    cudaDeviceGetAttribute(&n_sm[dev], cudaDevAttrMultiProcessorCount, dev);
    if (n_sm[dev] <= 0) n_sm[dev] = 148;
    attr_set[dev] = true;
  }
  const int tiles = n * ((oh + kTileRows - 1) / kTileRows);
  const int usable = n_sm[dev] - g_tsp_sm_reserve > 8 ? n_sm[dev] - g_tsp_sm_reserve : 8;
  const int grid = tiles < usable ? tiles : usable;
  conv_stem_wgrad_kernel<<<grid, kWgThreads, kWgSmemBytes, stream>>>(td, (const __nv_bfloat16*)x, (const __nv_bfloat16*)dy, n, h, w, oh, ow, dw, status);
  return TSP_LAUNCH_CHECK();
}

}  // extern "C"

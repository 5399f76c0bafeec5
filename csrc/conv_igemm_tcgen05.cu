// Implicit-GEMM convolutions (and the matching products of linear layers) on the 5th-generation tensor cores.
//
// Activations are channels-last bf16 ([N, H, W, C], C a multiple of 64), weights bf16 [Cout][kh][kw][Cin], square
// kernels of size 1 or 3, stride 1 or 2, padding (k - 1) / 2.  Three products, all with fp32 accumulation in TMEM:
//
//   forward    Y[p, co]  = sum_{tap, ci} X[p + tap, ci] * W[co, tap, ci]            (tsp_conv_fprop)
//   data grad  dX[p, ci] = sum_{tap, co} dY[p - tap, co] * W[co, tap, ci]           (tsp_conv_dgrad)
//   weight grad dW[co, tap, ci] += sum_p X[p + tap, ci] * dY[p, co]                 (tsp_conv_wgrad)
//
// No im2col buffer exists anywhere: an M tile is a BOX of output pixels (w x h x n, at most 128 of them) and the
// operand tile for one filter tap is that same box shifted by the tap's offset, fetched by ONE 4-D TMA tile load
// (cp.async.bulk.tensor.4d, 128-byte swizzle); rows that fall into the padding are zero-filled by the TMA unit.
// Stride 2 needs no strided traversal either: the input is addressed through four tensor maps, one per (row, column)
// parity, each an ordinary dense view with doubled pitches, and every tap reads exactly one of them.  A 1x1 stride-1
// convolution degenerates to a plain GEMM over the flattened pixels (box = 128 consecutive pixels).
//
// A 3x3 stride-1 convolution of an image at most 61 pixels wide does not fetch nine shifted boxes per channel block
// (nine trips through L2 for the same pixels): conv_halo_kernel loads the box ONCE with a one-pixel border
// ((w + 2) x (h + 2) pixels, border zero-filled by TMA), enumerates the accumulator rows in that bordered pitch, and
// the operand of tap (kh, kw) is the same shared-memory tile read from row kh * (w + 2) + kw on - a shifted start
// address in the matrix descriptor (whose base-offset field carries the swizzle phase of the shifted start).  The
// rows that correspond to border columns are computed and thrown away.
//
//   forward / data grad (conv_fwd_kernel): A = shifted pixel box [pixels x 64 channels], K-major; B = weight tile,
//     K-major for the forward ([co][tap, ci] rows) and MN-major for the data gradient (the same weight matrix read
//     as [co rows (K)][ci (N)] boxes, so no transposed copy of the weights is ever made).  The data gradient of a
//     stride-2 convolution runs once per output parity class with the taps that reach that class.  Epilogue: TMEM ->
//     registers -> bf16 -> shared memory -> 16-byte coalesced stores to the pixel addresses; optionally per-channel
//     sum / sum of squares of the rounded outputs (the statistics of the BatchNorm that follows), per view segment.
//   weight grad (conv_wgrad_kernel): both operands are pixel boxes as loaded, i.e. MN-major: M = (tap, ci) (two
//     64-channel boxes of the shifted input), N = co (BN / 64 boxes of dY), K = the box's pixels.  The pixel range is
//     split over CTAs and every CTA adds its partial tile into the fp32 gradient with red.global.add.f32 (coalesced
//     along ci), which is also what accumulates micro-batches.
//
// Roles per CTA (192 threads): warp 0 TMA producer, warp 1 MMA issuer + TMEM owner, warps 2-5 epilogue.  Persistent
// over tiles, shared-memory ring of 3-6 stages, two accumulator buffers in TMEM so the epilogue of tile i overlaps
// the MMAs of tile i + 1.  Every mbarrier wait is bounded: a wait that runs out writes a code into *status (1 producer,
// 2 MMA on operands, 3 epilogue, 4 MMA on a free accumulator), all roles leave their loops, TMEM is released.
//
// Reference call sites: every nn.Conv2d of the torchvision ResNets (`benchmarks/byol/models/resnet_base_network.py:60-77`,
// `benchmarks/soft_target/models/resnet.py`) and every nn.Linear backward of the ViT / BERT blocks and MLP heads
// (`benchmarks/moco-v3/vits.py`, `benchmarks/distilbert/bert.py:104-266`, `benchmarks/byol/models/mlp_head.py:4-26`),
// all library (cuDNN / cuBLAS) calls there.
#include <cuda.h>
#include <stdlib.h>

#include "tcgen05.cuh"
#include "tspipe_kernels.h"

namespace {

using namespace tc5;

constexpr int kThreads = 320;           // halo kernel: warp 0 TMA, warp 1 MMA, warps 2..9 epilogue (two per TMEM lane quarter)
constexpr int kWgThreads = 192;         // weight gradient: warp 0 TMA, warp 1 MMA, warps 2..5 epilogue
constexpr int kBoxBytes = 128 * 128;        // shared memory reserved per pixel box: 128 rows x 64 bf16
constexpr int kMaxTaps = 9;

struct Geom {
  int out_w, out_h, out_n;                  // extent of the pixel grid the tiles walk
  int box_w, box_h, box_n;                  // pixel box of one tile
  int tiles_w, tiles_h, tiles_n;
  int row_pitch;                            // accumulator rows per box row: box_w, or box_w + 2 in the halo kernel
  int pix;                                  // row_pitch * box_h * box_n  (<= 128): accumulator rows in use
  int halo_rows;                            // halo kernel: (box_w + 2) * (box_h + 2) rows fetched per channel block
  int b_resident;                           // halo kernel: the nine weight tiles are loaded once and stay
  int tma_store;                            // forward kernel, flat pixel grid: the epilogue writes with TMA stores
  int n_fastest;                            // tile index = m_tile * tiles_n + n_tile (else n_tile * tiles_m + m_tile)
  unsigned long long wait_ns;               // give-up time of every mbarrier wait
  // divisors that every role meets once or more per tile (a division by a number the compiler does not know is some thirty
  // instructions, and the nine of a tile were more than half of what an epilogue warp issued for it)
  tsp::FastDiv by_tiles_w, by_tiles_h, by_order, by_seg;      // by_order: channel tiles or pixel tiles, see split_tile
  int n_taps;
  int kc;                                   // channels per tap on the contraction side (forward) / on the M side (wgrad)
  int nc;                                   // channels on the N side
  int rows_per_seg;                         // statistics: pixels per segment, in walk order (n, h, w)
  int out_sn, out_sh, out_sw;               // output pitches of the pixel grid, in units of 8 elements
  int ldw;                                  // wgrad: row pitch of dW in elements
  int splits;                               // wgrad: pieces of the pixel range
  int tap_dw[kMaxTaps], tap_dh[kMaxTaps], tap_map[kMaxTaps], tap_col[kMaxTaps];
  int tap_off[kMaxTaps];                    // halo kernel: first shared-memory row of the tap's operand
};
struct ActMaps {
  CUtensorMap m[4];
};

// ADD: 0 no addend, 1 read by the epilogue's threads, 2 fetched by TMA (flat pixel grid): see add_epilogue
constexpr int kAddBufs = 4;
// GROUPS: epilogue warps per TMEM lane quarter
template <int BN, int ADD, int GROUPS>
struct FwdCfg {
  static constexpr int kABytes = kBoxBytes;
  static constexpr int kBBytes = BN * 128;
  static constexpr int kStageBytes = kABytes + kBBytes;
  static constexpr int kThreads = 64 + 128 * GROUPS;
  static constexpr int kStages = ADD == 2 ? (BN == 64 ? 4 : 2) : BN == 256 ? (GROUPS == 2 ? 4 : 3) : (BN == 128 && GROUPS == 4 ? 5 : 6);
  static constexpr int kGroup = GROUPS == 2 ? 2 : 1;        // stages released per tcgen05.commit (1024 -> 256 channels at 14 x 14,
  static constexpr int kGroups = kStages / kGroup;          // 64 images, B200: 13.4 us in twos, 14.5 one by one)
  static constexpr int kAccBufs = GROUPS == 2 || BN == 256 ? 2 : 4;
  static constexpr int kTmemCols = kAccBufs * BN;
  // 32-row x 128-byte staging blocks per epilogue warp
  static constexpr int kStoreBytes = 4 * GROUPS * (ADD == 2 ? kAddBufs : 1) * 32 * 128;
  static constexpr int kSmemBytes = kStages * kStageBytes + kStoreBytes + 1024 + 256 + (ADD == 2 ? 8 * 8 * kAddBufs : 0);
};

// Tiles are dealt to the CTAs in contiguous ranges (tile index = n_tile * tiles_m + m_tile): a CTA then stays on one
// block of output channels - one set of weights, one set of statistics accumulators - for nearly all of its tiles,
// and consecutive tiles are neighbouring pixel boxes.
__device__ __forceinline__ int tile_begin(int num_tiles, unsigned cta) {
  return (int)((long long)num_tiles * cta / gridDim.x);
}

// Split a tile index into (pixel tile, channel tile).  With statistics a CTA should stay on one channel block (one set
// of accumulators, few flushes): channel-major.  Without, channel tiles run fastest: the CTAs that run together share
// a pixel tile's input (fetched from DRAM once, then from L2) and sweep the weights, which stay in L2.
__device__ __forceinline__ void split_tile(const Geom& g, int t, int& tm, int& tn) {
  uint32_t rest;
  const uint32_t q = g.by_order.div((uint32_t)t, rest);
  tm = (int)(g.n_fastest ? q : rest);
  tn = (int)(g.n_fastest ? rest : q);
}
// Of a geometry that is complete, for `tiles_nn` channel tiles.
inline void set_divisors(Geom& g, int tiles_nn) {
  g.by_tiles_w = tsp::FastDiv(g.tiles_w);
  g.by_tiles_h = tsp::FastDiv(g.tiles_h);
  g.by_order = tsp::FastDiv(g.n_fastest ? tiles_nn : g.tiles_w * g.tiles_h * g.tiles_n);
  g.by_seg = tsp::FastDiv(g.rows_per_seg > 0 ? g.rows_per_seg : 1);
}

__device__ __forceinline__ void tile_origin(const Geom& g, int tm, int& w0, int& h0, int& n0) {
  uint32_t wb, hb;
  const uint32_t r = g.by_tiles_w.div((uint32_t)tm, wb), nb = g.by_tiles_h.div(r, hb);
  w0 = (int)wb * g.box_w;
  h0 = (int)hb * g.box_h;
  n0 = (int)nb * g.box_n;
}

// Epilogue warps (from 2 on) of the forward / data-gradient kernels.  A tile has `n_sub` accumulators of 128 rows (SUBS
// reserved per TMEM buffer); accumulator row p of the tile (p = 128 * sub + TMEM lane) is pixel
// (p % row_pitch, (p / row_pitch) % box_h, p / (row_pitch * box_h)) of the tile's box; rows in border columns, past
// the box or outside the image are not stored.  Warp w owns TMEM lanes 32 * (w % 4) .. + 31; the GROUPS warps that
// share a lane quarter split the tile's 64-channel blocks between them, and where there are fewer blocks than warps, a
// block's accumulators in turn.  Per unit: TMEM -> registers -> bf16
// -> swizzled shared memory (rows that are not stored are written as zeros) -> per-channel sums from shared memory
// (STATS) and coalesced 16-byte stores, 8 lanes per pixel.
// ADD: `addend` has the output's layout and is added to the rounded result, as the sum of two bf16 gradients would be.
template <int BN, int SUBS, int ACC_BUFS, int GROUPS, bool STATS, bool ADD>
__device__ __forceinline__ void fwd_epilogue(const Geom& g, int num_tiles, int n_sub, uint32_t tmem_base,
                                             uint64_t* tmem_full_bar, uint64_t* tmem_empty_bar, uint8_t* store_bufs,
                                             __nv_bfloat16* __restrict__ out,
                                             const __nv_bfloat16* __restrict__ addend, float* __restrict__ col_sums,
                                             int* __restrict__ status, int warp, int lane,
                                             const CUtensorMap* __restrict__ omap = nullptr) {
  const int quarter = warp & 3, group = (warp - 2) >> 2;
  const bool tma_out = !ADD && omap != nullptr && g.tma_store != 0;       // flat pixel grid: 32-row blocks go out as TMA stores
  uint8_t* buf = store_bufs + (warp - 2) * (32 * 128);
  uint32_t lt = 0;
  bool ok = true;
  constexpr int kBlocks = BN / 64;
  constexpr int kMine = kBlocks > GROUPS ? kBlocks / GROUPS : 1;        // this warp's 64-channel blocks of a tile
  constexpr int kShare = kBlocks < GROUPS ? GROUPS / kBlocks : 1;       // warps of a lane quarter that share a block
  auto block = [&](int j) -> int { return kShare > 1 ? group % kBlocks : j * GROUPS + group; };
  ColSums cs[kMine];
#pragma unroll
  for (int j = 0; j < kMine; ++j) cs[j].clear();
  int cur_c0 = -1, cur_seg = 0;
  auto flush_stats = [&]() {
    if (cur_c0 >= 0) {
      float* dst = col_sums + (int64_t)cur_seg * 2 * g.nc;
#pragma unroll
      for (int j = 0; j < kMine; ++j) {
        float s[2], q[2];
        cs[j].reduce(lane, s, q);
        const int col = cur_c0 + 64 * block(j) + ColSums::channel(lane);
        // (nc is a multiple of 64: col and col + 1 exist together)
        if (col < g.nc && (q[0] != 0.f || q[1] != 0.f)) {
          atomicAdd(dst + col, s[0]); atomicAdd(dst + g.nc + col, q[0]);
          atomicAdd(dst + col + 1, s[1]); atomicAdd(dst + g.nc + col + 1, q[1]);
        }
        cs[j].clear();
      }
    }
  };
  // the lane's pixel of each accumulator within the box, far outside the image for a row that is none
  int3 in_box[SUBS];
#pragma unroll
  for (int sub = 0; sub < SUBS; ++sub) {
    const int p = sub * 128 + quarter * 32 + lane, r2 = p / g.row_pitch;
    in_box[sub] = make_int3(p - r2 * g.row_pitch, r2 % g.box_h, r2 / g.box_h);
    if (p >= g.pix || in_box[sub].x >= g.box_w) in_box[sub].x = 1 << 30;
  }
  const int t_begin = tile_begin(num_tiles, blockIdx.x), t_end = tile_begin(num_tiles, blockIdx.x + 1);
  for (int t = t_begin; t < t_end && ok; ++t, ++lt) {
    int w0, h0, n0, tm, tn;
    split_tile(g, t, tm, tn);
    tile_origin(g, tm, w0, h0, n0);
    const int c0 = tn * BN;
    const uint32_t acc = lt % ACC_BUFS, use = lt / ACC_BUFS;
    if (STATS) {
      const int seg = (int)g.by_seg.div((uint32_t)((n0 * g.out_h + h0) * g.out_w + w0));       // (fewer than 2^31 pixels)
      if (c0 != cur_c0 || seg != cur_seg) { flush_stats(); cur_c0 = c0; cur_seg = seg; }
    }
    // a lane's pixel and where it is stored (units of 8 elements), -1 for rows that are not stored
    auto pixel_off = [&](int sub) -> int {
      const int w = w0 + in_box[sub].x, h = h0 + in_box[sub].y, n = n0 + in_box[sub].z;
      return w < g.out_w && h < g.out_h && n < g.out_n ? n * g.out_sn + h * g.out_sh + w * g.out_sw : -1;
    };
    const int pc = lane & 7;
    auto takes = [&](int sub) -> bool { return kShare == 1 || (int)((lt * n_sub + sub) % kShare) == group / kBlocks; };
    constexpr bool kEarly = ADD && SUBS == 1;
    // ADD: the addend in the layout of the stores below.  One accumulator: the whole tile's is requested before the
    // accumulator is waited for, so that its way from memory overlaps the products.
    uint4 add[ADD && kEarly ? kMine : 1][ADD ? 8 : 1];
    auto load_add = [&](uint4 (&dst)[ADD ? 8 : 1], int row_off, int col) {
      if constexpr (ADD) {
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const int off = __shfl_sync(0xffffffffu, row_off, 4 * k + (lane >> 3));
          dst[k] = make_uint4(0u, 0u, 0u, 0u);
          if (off >= 0) dst[k] = __ldcs(reinterpret_cast<const uint4*>(addend + ((int64_t)off << 3) + col + pc * 8));
        }
      }
    };
    if constexpr (kEarly) {
      const int row_off = pixel_off(0);
#pragma unroll
      for (int j = 0; j < kMine; ++j)
        if (takes(0) && c0 + 64 * block(j) < g.nc) load_add(add[j], row_off, c0 + 64 * block(j));
    }
    ok = mbar_wait_warp(tmem_full_bar + acc, use & 1, status, 3, g.wait_ns, lane);
    if (!ok) break;
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
    for (int sub = 0; sub < SUBS; ++sub) {
      if (sub < n_sub && takes(sub)) {
        const int row_off = pixel_off(sub);
#pragma unroll
        for (int b = 0; b < kMine; ++b) {
          const int col = c0 + 64 * block(b);
          if (col < g.nc) {
            if constexpr (ADD && !kEarly) load_add(add[0], row_off, col);
            // (four warps per quarter have half the registers each, and each other to fill the waits)
            constexpr int kPart = GROUPS > 2 ? 32 : 64;
            uint32_t r[kPart];
            const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + (acc * SUBS + sub) * BN + (uint32_t)(64 * block(b));
            uint8_t* my_row = buf + lane * 128;
            const bool keep = row_off >= 0;
#pragma unroll
            for (int at = 0; at < 64; at += kPart) {
              tmem_ld_32x32_issue(taddr + at, r);
              if constexpr (kPart == 64) tmem_ld_32x32_issue(taddr + 32, r + 32);
              tmem_ld_wait();
              if (tma_out && at == 0) {             // the previous block's store has finished reading the staging buffer
                if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
                __syncwarp();
              }
#pragma unroll
              for (int j = 0; j < kPart / 8; ++j) {         // 16-byte piece j of this row sits at piece (j ^ (row & 7))
                uint4 q = make_uint4(0u, 0u, 0u, 0u);
                if (keep) {
                  q.x = pack_bf16x2(__uint_as_float(r[8 * j + 0]), __uint_as_float(r[8 * j + 1]));
                  q.y = pack_bf16x2(__uint_as_float(r[8 * j + 2]), __uint_as_float(r[8 * j + 3]));
                  q.z = pack_bf16x2(__uint_as_float(r[8 * j + 4]), __uint_as_float(r[8 * j + 5]));
                  q.w = pack_bf16x2(__uint_as_float(r[8 * j + 6]), __uint_as_float(r[8 * j + 7]));
                }
                *reinterpret_cast<uint4*>(my_row + (((at / 8 + j) ^ (lane & 7)) << 4)) = q;
              }
            }
            __syncwarp();
            if (tma_out) {
              asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
              __syncwarp();
              if (lane == 0) tma_store_2d(omap, buf, col, w0 + sub * 128 + quarter * 32);   // rows past the end are clipped
            } else {
              // coalesced stores: 8 lanes write the 128 bytes of one pixel's channel block, 4 pixels per instruction
#pragma unroll
              for (int k = 0; k < 8; ++k) {
                const int rr = 4 * k + (lane >> 3);
                const int off = __shfl_sync(0xffffffffu, row_off, rr);
                uint4 q = *reinterpret_cast<const uint4*>(buf + rr * 128 + ((pc ^ (rr & 7)) << 4));
                if constexpr (ADD) {
                  __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&q);
                  const __nv_bfloat162* a = reinterpret_cast<const __nv_bfloat162*>(&add[kEarly ? b : 0][k]);
#pragma unroll
                  for (int e = 0; e < 4; ++e) h[e] = __hadd2(h[e], a[e]);
                }
                if (off >= 0) *reinterpret_cast<uint4*>(out + ((int64_t)off << 3) + col + pc * 8) = q;
              }
              __syncwarp();
            }
            // (the block's stores are on their way: the sums overlap them)
            if (STATS) cs[b].add(buf, lane);         // of the rounded block (rows that are not stored hold zeros)
          }
        }
      }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncwarp();
    if (lane == 0) mbar_arrive(tmem_empty_bar + acc);
  }
  if (tma_out) {
    if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");     // staging buffer free, stores complete
    __syncwarp();
  }
  if (STATS) {
    // the last sums go through the staging buffer: the CTA adds its warps' up before they leave (flush_cta_stats)
    float* st = reinterpret_cast<float*>(buf);
#pragma unroll
    for (int j = 0; j < kMine; ++j) {
      float s[2], q[2];
      cs[j].reduce(lane, s, q);
      *reinterpret_cast<float2*>(st + j * 128 + ColSums::channel(lane)) = make_float2(s[0], s[1]);
      *reinterpret_cast<float2*>(st + j * 128 + 64 + ColSums::channel(lane)) = make_float2(q[0], q[1]);
    }
    if (lane == 0) { st[512] = __int_as_float(ok ? cur_c0 : -1); st[513] = __int_as_float(cur_seg); }
  }
}

// The sums that the epilogue warps left in their staging buffers, added up and sent as one addition per channel and CTA,
// lane = channel.  Additions to one 32-byte sector of memory are serialised at some 15 ns each: with every warp sending
// its own, two instructions a sector, the 148 CTAs of a convolution with 64 to 256 output channels queued for up to
// 30 us at their end.  The convolutions of a ResNet-50
// forward over 64 images, B200: 1354 us then, 1210 now.
template <int BN, int GROUPS>
__device__ __forceinline__ void flush_cta_stats(const Geom& g, const uint8_t* store_bufs, float* __restrict__ col_sums) {
  constexpr int kBlocks = BN / 64, kShare = kBlocks < GROUPS ? GROUPS / kBlocks : 1;        // as in fwd_epilogue
  auto part = [&](int w) { return reinterpret_cast<const float*>(store_bufs + w * (32 * 128)); };
  const int c0 = __float_as_int(part(0)[512]), seg = __float_as_int(part(0)[513]);
  for (int w = 1; w < 4 * GROUPS; ++w)            // all warps walk the same tiles; after a wait that ran out nothing is added
    if (__float_as_int(part(w)[512]) != c0) return;
  if (c0 < 0) return;
  float* dst = col_sums + (int64_t)seg * 2 * g.nc;
  for (int p = threadIdx.x; p < 2 * BN; p += 64 + 128 * GROUPS) {
    const int half = p / BN, col = p % BN, i = col >> 6;
    const int group = kShare > 1 ? i : i % GROUPS, at = (kShare > 1 ? 0 : i / GROUPS) * 128 + half * 64 + (col & 63);
    if (c0 + col >= g.nc) continue;
    float v = 0.f;
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
      for (int k = 0; k < kShare; ++k) v += part((group + k * kBlocks) * 4 + q)[at];
    atomicAdd(dst + half * g.nc + c0 + col, v);
  }
}

// Epilogue of a data gradient with an addend on a flat pixel grid.  Per warp a ring of staging blocks: the addend's block of
// the third unit from here is on its way by TMA while this unit's sum is formed in its block and leaves it by TMA, so that
// 96 KB per SM are in flight whatever the tile is waiting for.  Read by the threads instead, one tile ahead in registers, the
// gradient of [256, 56, 56, 256] took 223 us, 157 this way (141 at the rate of a copy).
template <int BN>
__device__ __forceinline__ void add_epilogue(const Geom& g, int num_tiles, uint32_t tmem_base,
                                             uint64_t* tmem_full_bar, uint64_t* tmem_empty_bar, uint8_t* store_bufs,
                                             uint64_t* add_bars, const CUtensorMap* __restrict__ omap,
                                             const CUtensorMap* __restrict__ amap, int* __restrict__ status, int warp, int lane) {
  const int quarter = warp & 3, group = (warp - 2) >> 2;
  constexpr int kBlocks = BN / 64, kMine = (kBlocks + 1) / 2;         // 64-channel blocks of a tile, and of them this warp's
  uint8_t* bufs = store_bufs + (warp - 2) * kAddBufs * (32 * 128);
  uint64_t* bars = add_bars + (warp - 2) * kAddBufs;
  const int t_begin = tile_begin(num_tiles, blockIdx.x), t_end = tile_begin(num_tiles, blockIdx.x + 1);
  const bool idle = kBlocks == 1 && group == 1;
  const int units = idle ? 0 : (t_end - t_begin) * kMine;
  auto place = [&](int u, int& col, int& row) {
    int w0, h0, n0, tm, tn;
    split_tile(g, t_begin + u / kMine, tm, tn);
    tile_origin(g, tm, w0, h0, n0);
    col = tn * BN + 64 * (kBlocks == 1 ? 0 : 2 * (u % kMine) + group);
    row = w0 + quarter * 32;
  };
  auto fetch = [&](int u) {                     // (a block past the last channel or pixel reads as zeros)
    int col, row;
    place(u, col, row);
    uint64_t* bar = bars + u % kAddBufs;
    mbar_expect_tx(bar, 32 * 128);
    tma_load_2d(bufs + u % kAddBufs * (32 * 128), amap, bar, col, row);
  };
  if (lane == 0)
    for (int u = 0; u < kAddBufs - 1 && u < units; ++u) fetch(u);
  bool ok = true;
  for (int t = t_begin, lt = 0; t < t_end && ok; ++t, ++lt) {
    const uint32_t acc = lt & 1, use = lt >> 1;
    ok = mbar_wait_warp(tmem_full_bar + acc, use & 1, status, 3, g.wait_ns, lane);
    if (!ok) break;
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
    for (int j = 0; j < kMine; ++j) {
      if (idle) continue;
      const int u = lt * kMine + j;
      uint8_t* buf = bufs + u % kAddBufs * (32 * 128);
      uint32_t r[64];
      const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + acc * BN + (uint32_t)(64 * (kBlocks == 1 ? 0 : 2 * j + group));
      tmem_ld_32x32_issue(taddr, r);
      tmem_ld_32x32_issue(taddr + 32, r + 32);
      ok = mbar_wait_warp(bars + u % kAddBufs, (u / kAddBufs) & 1, status, 3, g.wait_ns, lane);
      tmem_ld_wait();
      if (!ok) break;
      uint8_t* my_row = buf + lane * 128;
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        uint4* at = reinterpret_cast<uint4*>(my_row + ((q ^ (lane & 7)) << 4));
        uint4 v = *at;
        __nv_bfloat162* a = reinterpret_cast<__nv_bfloat162*>(&v);
#pragma unroll
        for (int e = 0; e < 4; ++e)
          a[e] = __hadd2(__floats2bfloat162_rn(__uint_as_float(r[8 * q + 2 * e]), __uint_as_float(r[8 * q + 2 * e + 1])), a[e]);
        *at = v;
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) {
        int col, row;
        place(u, col, row);
        if (col < g.nc && row < g.out_w) tma_store_2d(omap, buf, col, row);             // rows past the end are clipped
        else asm volatile("cp.async.bulk.commit_group;" ::: "memory");
        // the block of unit u - 1 is free once its store has read it: the next to be fetched takes it
        asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
        if (u + kAddBufs - 1 < units) fetch(u + kAddBufs - 1);
      }
      __syncwarp();
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncwarp();
    if (lane == 0) mbar_arrive(tmem_empty_bar + acc);
  }
  if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  __syncwarp();
}

// ---------------------------------------------------------------------------------------------------------------
// forward / data gradient
// ---------------------------------------------------------------------------------------------------------------
template <int BN, bool B_MN, bool STATS, int ADD, int GROUPS>
__global__ void __launch_bounds__(FwdCfg<BN, ADD, GROUPS>::kThreads, 1)
conv_fwd_kernel(const __grid_constant__ ActMaps amaps, const __grid_constant__ CUtensorMap wmap,
                const __grid_constant__ CUtensorMap omap, const __grid_constant__ CUtensorMap addmap,
                const __grid_constant__ Geom g, __nv_bfloat16* __restrict__ out,
                const __nv_bfloat16* __restrict__ addend, float* __restrict__ col_sums, int* __restrict__ status) {
  extern __shared__ uint8_t smem_raw[];
  using C = FwdCfg<BN, ADD, GROUPS>;
  uint8_t* tiles = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint8_t* store_bufs = tiles + C::kStages * C::kStageBytes;
  uint64_t* bars = (uint64_t*)(store_bufs + C::kStoreBytes);
  uint64_t* full_bar = bars;
  uint64_t* empty_bar = bars + C::kStages;
  uint64_t* tmem_full_bar = bars + 2 * C::kStages;
  uint64_t* tmem_empty_bar = tmem_full_bar + C::kAccBufs;
  uint32_t* tmem_slot = (uint32_t*)(tmem_empty_bar + C::kAccBufs);
  uint64_t* add_bars = tmem_empty_bar + C::kAccBufs + 1;             // [8 warps][kAddBufs]  addend -> epilogue (ADD == 2)

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tiles_m = g.tiles_w * g.tiles_h * g.tiles_n, tiles_nn = (g.nc + BN - 1) / BN;
  const int num_tiles = tiles_m * tiles_nn;
  const int kcb = g.kc >> 6;
  const int num_kb = g.n_taps * kcb;

  if (threadIdx.x == 0) {
    for (int s = 0; s < C::kStages; ++s) {
      mbar_init(full_bar + s, 1);
      mbar_init(empty_bar + s, 1);
    }
    for (int a = 0; a < C::kAccBufs; ++a) {
      mbar_init(tmem_full_bar + a, 1);
      mbar_init(tmem_empty_bar + a, 4 * GROUPS);
    }
    if (ADD == 2)
      for (int i = 0; i < 8 * kAddBufs; ++i) mbar_init(add_bars + i, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&amaps.m[0]) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&wmap) : "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"((uint32_t)C::kTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = *tmem_slot;
  tsp::wait_for_previous();
  addend = tsp::written(addend);

  if (warp == 0) {
    // ---------------- TMA producer ----------------
    if (lane == 0) {
      uint32_t it = 0;
      bool ok = true;
      const uint32_t tx = (uint32_t)(g.pix * 128 + C::kBBytes);     // a box is written in full, zero fill included
      for (int t = tile_begin(num_tiles, blockIdx.x); t < tile_begin(num_tiles, blockIdx.x + 1) && ok; ++t) {
        int w0, h0, n0, tm, tn;
        split_tile(g, t, tm, tn);
        tile_origin(g, tm, w0, h0, n0);
        const int c0 = tn * BN;
        for (int tap = 0; tap < g.n_taps && ok; ++tap) {
          const CUtensorMap* am = &amaps.m[g.tap_map[tap]];
          const int xw = w0 + g.tap_dw[tap], xh = h0 + g.tap_dh[tap], wcol = g.tap_col[tap];
          for (int cb = 0; cb < kcb; ++cb, ++it) {
            const int s = it % C::kStages;
            if (it % C::kGroup == 0) {              // first stage of a group: the whole group must have been released
              const uint32_t grp = (it / C::kGroup) % C::kGroups, round = (it / C::kGroup) / C::kGroups;
              if (round > 0 && !mbar_wait_parked(empty_bar + grp, (round - 1) & 1, status, 1, g.wait_ns)) { ok = false; break; }
            }
            uint8_t* a_dst = tiles + s * C::kStageBytes;
            uint8_t* b_dst = a_dst + C::kABytes;
            mbar_expect_tx(full_bar + s, tx);
            tma_load_4d(a_dst, am, full_bar + s, cb * 64, xw, xh, n0);
            if constexpr (!B_MN) {
              tma_load_2d(b_dst, &wmap, full_bar + s, wcol + cb * 64, c0);       // [BN rows (co)][64 (tap, ci)]
            } else {
#pragma unroll
              for (int j = 0; j < BN / 64; ++j)                                  // [64 rows (co)][64 (tap, ci)] each
                tma_load_2d(b_dst + j * 8192, &wmap, full_bar + s, wcol + c0 + j * 64, cb * 64);
            }
          }
        }
      }
      tsp::let_next_start();
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer ----------------
    {
      const bool issuer = tc5::elect_one();
      auto arrived = [&](uint64_t* bar, uint32_t parity, int code) -> bool {      // the same for the warp
        return __all_sync(0xffffffffu, tc5::mbar_wait(bar, parity, status, code, g.wait_ns)) != 0;
      };
      constexpr uint32_t idesc = make_idesc(128, BN, false, B_MN);
      const uint32_t tiles_addr = smem_u32(tiles);
      uint32_t it = 0, lt = 0;
      // The next operands and the next accumulator, looked at ahead (mbar_over), where the contraction is long: 64 images, B200,
      // 512 -> 512 3x3 at 7 x 7 26.2 us without, 23.7 with, 512 -> 128 1x1 at 28 x 28 (8 blocks) 18.4 and 18.0, 256 -> 256 3x3 of
      // stride 2 at 28 x 28 29.5 and 25.1, 256 -> 512 3x3 of stride 2 at 56 x 56 119.4 and 120.5; with 4 blocks 256 -> 512 1x1 of stride
      // 2 at 56 x 56 27.0 and 27.8.
      const bool ahead = num_kb >= 8;
      bool ok = true, there = false, room = false;
      for (int t = tile_begin(num_tiles, blockIdx.x); t < tile_begin(num_tiles, blockIdx.x + 1) && ok; ++t, ++lt) {
        const uint32_t acc = lt % C::kAccBufs, use = lt / C::kAccBufs;
        if (use > 0) {
          if (!__all_sync(0xffffffffu, room)) ok = arrived(tmem_empty_bar + acc, (use - 1) & 1, 4);
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        }
        const uint32_t d_tmem = tmem_base + acc * BN;
        uint32_t accum = 0u;
        for (int kb = 0; kb < num_kb; ++kb, ++it) {
          const int s = it % C::kStages;
          const uint32_t round = it / C::kStages;
          if (!__all_sync(0xffffffffu, there)) ok = arrived(full_bar + s, round & 1, 2);
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          there = ahead && mbar_over(full_bar + (it + 1) % C::kStages, ((it + 1) / C::kStages) & 1);
          if (ahead && kb == num_kb - 1)
            room = lt + 1 >= (uint32_t)C::kAccBufs &&
                   mbar_over(tmem_empty_bar + (lt + 1) % C::kAccBufs, ((lt + 1) / C::kAccBufs - 1) & 1);
          const uint32_t a_addr = tiles_addr + s * C::kStageBytes;
          const uint32_t a_lo = desc_lo_k_major(a_addr);
          const uint32_t b_lo = B_MN ? desc_lo_mn_major(a_addr + C::kABytes, 8192) : desc_lo_k_major(a_addr + C::kABytes);
#pragma unroll
          for (int kk = 0; kk < 4; ++kk) {          // 16 along K: +32 bytes in a K-major row, +2048 bytes (16 rows) MN-major
            if (issuer) umma_bf16_lo(d_tmem, a_lo + 2 * kk, b_lo + (B_MN ? 128 * kk : 2 * kk), idesc, accum);
            accum = 1u;
          }
          if (issuer && it % C::kGroup == C::kGroup - 1) umma_commit(empty_bar + (it / C::kGroup) % C::kGroups);
        }
        if (issuer) umma_commit(tmem_full_bar + acc);
      }
    }
  } else {
    if constexpr (ADD == 2)
      add_epilogue<BN>(g, num_tiles, tmem_base, tmem_full_bar, tmem_empty_bar, store_bufs, add_bars, &omap, &addmap,
                       status, warp, lane);
    else
      fwd_epilogue<BN, 1, C::kAccBufs, GROUPS, STATS, ADD == 1>(g, num_tiles, 1, tmem_base, tmem_full_bar,
                                                                       tmem_empty_bar, store_bufs, out, addend, col_sums, status, warp,
                                                                       lane, &omap);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (STATS) flush_cta_stats<BN, GROUPS>(g, store_bufs, col_sums);
  if (warp == 1) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)C::kTmemCols)
                 : "memory");
  }
}

// ---------------------------------------------------------------------------------------------------------------
// 3x3, stride 1: forward / data gradient with the bordered pixel box resident in shared memory
// ---------------------------------------------------------------------------------------------------------------
template <int BN>
struct HaloCfg {
  static constexpr int kARows = 384;                          // bordered box: up to 256 accumulator rows + 2 rows + 2
  static constexpr int kABytes = kARows * 128;
  static constexpr int kAStages = 2;
  static constexpr int kBBytes = BN * 128;                    // weights of one tap and one 64-channel block
  static constexpr int kBStages = BN == 64 ? 9 : (BN == 128 ? 6 : 3);
  static constexpr int kBGroup = BN == 256 ? 1 : 3;           // weight stages released per tcgen05.commit
  static constexpr int kBGroups = kBStages / kBGroup;
  static constexpr int kAccBufs = BN == 256 ? 1 : 2;          // TMEM: kAccBufs x 2 accumulators x BN columns <= 512
  static constexpr int kTmemCols = kAccBufs * 2 * BN;
  static constexpr int kStoreBytes = 8 * 32 * 128;
  static constexpr int kSmemBytes = kAStages * kABytes + kBStages * kBBytes + kStoreBytes + 1024 + 512;
};

// The operand of tap (kh, kw) is the bordered box read from row tap_off = kh * pitch + kw on: a start address that is
// not 1024-byte aligned.  The tensor core applies the 128-byte swizzle to the bits of the absolute shared-memory
// address, as TMA did when it wrote the tile, so the shifted start needs nothing beyond its address (the descriptor's
// base-offset field stays 0; setting it to the start's phase gives wrong products - measured).
// One tile = a bordered box of up to 256 accumulator rows (two 128-row accumulators that share every weight tile).
// g.b_resident: all weight tiles of the problem (9 taps, one channel block, one N tile) fit the weight ring; they are
// loaded once and stay.  With 64 output channels a product takes the tensor pipe 63 clocks (its shared-memory reads), so
// the issuing thread is the bound: the taps are unrolled without the ring's waits, and one commit per tile tells the
// epilogue and, in place of a_empty, the producer.  256 images of 56 x 56, B200: forward with statistics
// 119 us with the ring's loop, 96 this way, 77 with the products issued by a converged warp; data gradient 110, 94 and 72.
template <int BN, bool B_MN, bool STATS, bool ADD>
__global__ void __launch_bounds__(kThreads, 1)
conv_halo_kernel(const __grid_constant__ CUtensorMap amap, const __grid_constant__ CUtensorMap wmap,
                 const __grid_constant__ Geom g, __nv_bfloat16* __restrict__ out,
                 const __nv_bfloat16* __restrict__ addend, float* __restrict__ col_sums, int* __restrict__ status) {
  extern __shared__ uint8_t smem_raw[];
  using C = HaloCfg<BN>;
  uint8_t* a_tiles = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint8_t* b_tiles = a_tiles + C::kAStages * C::kABytes;
  uint8_t* store_bufs = b_tiles + C::kBStages * C::kBBytes;
  uint64_t* bars = (uint64_t*)(store_bufs + C::kStoreBytes);
  uint64_t* a_full = bars;
  uint64_t* a_empty = a_full + C::kAStages;
  uint64_t* b_full = a_empty + C::kAStages;
  uint64_t* b_empty = b_full + C::kBStages;
  uint64_t* tmem_full_bar = b_empty + C::kBStages;
  uint64_t* tmem_empty_bar = tmem_full_bar + 2;
  uint32_t* tmem_slot = (uint32_t*)(tmem_empty_bar + 2);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tiles_m = g.tiles_w * g.tiles_h * g.tiles_n, tiles_nn = (g.nc + BN - 1) / BN;
  const int num_tiles = tiles_m * tiles_nn;
  const int kcb = g.kc >> 6;
  const int n_sub = (g.pix + 127) >> 7;
  const bool resident = g.b_resident != 0;
  // (resident: one channel block, so unit = tile, and stage u % 2 of the boxes goes with accumulator buffer u % 2)
  constexpr bool kMayReside = C::kBStages >= 9 && C::kAccBufs == C::kAStages;
  uint64_t* box_free = kMayReside && resident ? tmem_full_bar : a_empty;

  // Rows of an A stage past the bordered box are never written by TMA but are read for accumulator rows that are
  // thrown away; they are zeroed once so that those rows stay finite.
  {
    uint4* p = reinterpret_cast<uint4*>(a_tiles);
    for (int i = threadIdx.x; i < C::kAStages * C::kABytes / 16; i += kThreads) p[i] = make_uint4(0, 0, 0, 0);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (threadIdx.x == 0) {
    for (int s = 0; s < C::kAStages; ++s) { mbar_init(a_full + s, 1); mbar_init(a_empty + s, 1); }
    for (int s = 0; s < C::kBStages; ++s) { mbar_init(b_full + s, 1); mbar_init(b_empty + s, 1); }
    for (int a = 0; a < 2; ++a) { mbar_init(tmem_full_bar + a, 1); mbar_init(tmem_empty_bar + a, 8); }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&amap) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&wmap) : "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"((uint32_t)C::kTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = *tmem_slot;
  tsp::wait_for_previous();
  addend = tsp::written(addend);
  const int t_first = tile_begin(num_tiles, blockIdx.x), my_tiles = tile_begin(num_tiles, blockIdx.x + 1) - t_first;

  if (warp == 0) {
    // ---------------- TMA producer: one bordered box per (tile, channel block), nine weight tiles after it; the box
    // of the NEXT channel block is requested before the weight tiles of the current one ----------------
    if (lane == 0) {
      const int units = my_tiles * kcb;
      uint32_t ib = 0;
      bool ok = true;
      auto load_a = [&](int u) -> bool {
        const int t = t_first + u / kcb, cb = u % kcb;
        int w0, h0, n0, tm, tn;
        split_tile(g, t, tm, tn);
        tile_origin(g, tm, w0, h0, n0);
        const int s = u % C::kAStages;
        const uint32_t round = (uint32_t)u / C::kAStages;
        if (round > 0 && !mbar_wait_parked(box_free + s, (round - 1) & 1, status, 1, g.wait_ns)) return false;
        mbar_expect_tx(a_full + s, (uint32_t)g.halo_rows * 128u);
        tma_load_4d(a_tiles + s * C::kABytes, &amap, a_full + s, cb * 64, w0 - 1, h0 - 1, n0);
        return true;
      };
      if (units > 0) ok = load_a(0);
      for (int u = 0; u < units && ok; ++u) {
        if (u + 1 < units && !load_a(u + 1)) { ok = false; break; }
        if (resident && u > 0) continue;
        const int t = t_first + u / kcb, cb = u % kcb;
        int tm, tn;
        split_tile(g, t, tm, tn);
        const int c0 = tn * BN;
        for (int tap = 0; tap < 9; ++tap, ++ib) {
          const int s = ib % C::kBStages;
          if (ib % C::kBGroup == 0) {
            const uint32_t grp = (ib / C::kBGroup) % C::kBGroups, round = (ib / C::kBGroup) / C::kBGroups;
            if (round > 0 && !mbar_wait_parked(b_empty + grp, (round - 1) & 1, status, 1, g.wait_ns)) { ok = false; break; }
          }
          uint8_t* b_dst = b_tiles + s * C::kBBytes;
          mbar_expect_tx(b_full + s, (uint32_t)C::kBBytes);
          if constexpr (!B_MN) {
            tma_load_2d(b_dst, &wmap, b_full + s, g.tap_col[tap] + cb * 64, c0);
          } else {
#pragma unroll
            for (int j = 0; j < BN / 64; ++j)
              tma_load_2d(b_dst + j * 8192, &wmap, b_full + s, g.tap_col[tap] + c0 + j * 64, cb * 64);
          }
        }
      }
      tsp::let_next_start();
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer ----------------
    {
      const bool issuer = tc5::elect_one();
      auto arrived = [&](uint64_t* bar, uint32_t parity, int code) -> bool {      // the same for the warp
        return __all_sync(0xffffffffu, tc5::mbar_wait(bar, parity, status, code, g.wait_ns)) != 0;
      };
      constexpr uint32_t idesc = make_idesc(128, BN, false, B_MN);
      const uint32_t a_addr0 = smem_u32(a_tiles), b_addr0 = smem_u32(b_tiles);
      uint32_t ia = 0, ib = 0;
      bool ok = true;
      for (int lt = 0; lt < my_tiles && ok; ++lt) {
        const uint32_t acc = (uint32_t)lt % C::kAccBufs, use = (uint32_t)lt / C::kAccBufs;
        if (use > 0) {
          ok = arrived(tmem_empty_bar + acc, (use - 1) & 1, 4);
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        }
        const uint32_t d_tmem = tmem_base + acc * 2 * BN;
        uint32_t accum = 0u;
        for (int cb = 0; cb < kcb && ok; ++cb, ++ia) {
          const int sa = ia % C::kAStages;
          ok = arrived(a_full + sa, (ia / C::kAStages) & 1, 2);
          if (!ok) break;
          const uint32_t a_lo0 = desc_lo_k_major(a_addr0 + sa * C::kABytes);
          if constexpr (kMayReside) {
            if (resident) {
              if (ia == 0)
                for (int tap = 0; tap < 9 && ok; ++tap) ok = arrived(b_full + tap, 0u, 2);
              if (!ok) break;
              asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
              const uint32_t b_lo0 = B_MN ? desc_lo_mn_major(b_addr0, 8192) : desc_lo_k_major(b_addr0);
              auto products = [&](uint32_t d, uint32_t a_first) {
#pragma unroll
                for (int tap = 0; tap < 9; ++tap)
#pragma unroll
                  for (int kk = 0; kk < 4; ++kk)
                    if (issuer) umma_bf16_lo(d, a_first + 8 * g.tap_off[tap] + 2 * kk,
                                 b_lo0 + tap * (C::kBBytes >> 4) + (B_MN ? 128 * kk : 2 * kk), idesc, tap + kk > 0 ? 1u : 0u);
              };
              products(d_tmem, a_lo0);
              if (n_sub > 1) products(d_tmem + BN, a_lo0 + 1024);   // second accumulator: 128 rows further on
              continue;
            }
          }
          for (int tap = 0; tap < 9; ++tap, ++ib) {
            const int sb = (int)(ib % C::kBStages);
            ok = arrived(b_full + sb, (ib / C::kBStages) & 1, 2);
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t b_addr = b_addr0 + sb * C::kBBytes;
            const uint32_t b_lo = B_MN ? desc_lo_mn_major(b_addr, 8192) : desc_lo_k_major(b_addr);
            const uint32_t a_lo = a_lo0 + 8 * g.tap_off[tap];        // one row = 128 bytes = 8 address units
#pragma unroll
            for (int kk = 0; kk < 4; ++kk)
              if (issuer) umma_bf16_lo(d_tmem, a_lo + 2 * kk, b_lo + (B_MN ? 128 * kk : 2 * kk), idesc, kk == 0 ? accum : 1u);
            if (n_sub > 1) {
#pragma unroll
              for (int kk = 0; kk < 4; ++kk)                         // second accumulator: 128 rows further on
                if (issuer) umma_bf16_lo(d_tmem + BN, a_lo + 1024 + 2 * kk, b_lo + (B_MN ? 128 * kk : 2 * kk), idesc,
                             kk == 0 ? accum : 1u);
            }
            accum = 1u;
            if (issuer && ib % C::kBGroup == C::kBGroup - 1) umma_commit(b_empty + (ib / C::kBGroup) % C::kBGroups);
          }
          if (issuer && ok) umma_commit(a_empty + sa);
        }
        if (issuer) umma_commit(tmem_full_bar + acc);
      }
    }
  } else {
    fwd_epilogue<BN, 2, C::kAccBufs, 2, STATS, ADD>(g, num_tiles, n_sub, tmem_base, tmem_full_bar, tmem_empty_bar,
                                                 store_bufs, out, addend, col_sums, status, warp, lane);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (STATS) flush_cta_stats<BN, 2>(g, store_bufs, col_sums);
  if (warp == 1) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)C::kTmemCols)
                 : "memory");
  }
}

// ---------------------------------------------------------------------------------------------------------------
// weight gradient
// ---------------------------------------------------------------------------------------------------------------
template <int BN>
struct WgCfg {
  static constexpr int kBoxRows = BN == 256 ? 64 : 128;         // pixels per box (the K extent of one stage)
  static constexpr int kBox = kBoxRows * 128;                   // bytes reserved per box
  static constexpr int kABytes = 2 * kBox;                      // two 64-channel boxes of the shifted input (M = 128)
  static constexpr int kBBytes = (BN / 64) * kBox;              // BN / 64 boxes of dY
  static constexpr int kStageBytes = kABytes + kBBytes;
  static constexpr int kStages = BN == 128 ? 3 : 4;
  static constexpr int kGroup = BN == 128 ? 1 : 2;              // stages released per tcgen05.commit
  static constexpr int kGroups = kStages / kGroup;
  static constexpr int kTmemCols = 2 * BN;
  static constexpr int kSmemBytes = kStages * kStageBytes + 1024 + 256;
};

template <int BN>
__global__ void __launch_bounds__(kWgThreads, 1)
conv_wgrad_kernel(const __grid_constant__ ActMaps xmaps, const __grid_constant__ CUtensorMap dymap,
                  const __grid_constant__ Geom g, float* __restrict__ dw, int* __restrict__ status) {
  extern __shared__ uint8_t smem_raw[];
  using C = WgCfg<BN>;
  uint8_t* tiles = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint64_t* bars = (uint64_t*)(tiles + C::kStages * C::kStageBytes);
  uint64_t* full_bar = bars;
  uint64_t* empty_bar = bars + C::kStages;
  uint64_t* tmem_full_bar = bars + 2 * C::kStages;
  uint64_t* tmem_empty_bar = bars + 2 * C::kStages + 2;
  uint32_t* tmem_slot = (uint32_t*)(bars + 2 * C::kStages + 4);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int kcb = g.kc >> 6;
  const int m_blocks = g.n_taps * kcb;                       // 64-wide blocks of the (tap, ci) index
  const int m_tiles = (m_blocks + 1) >> 1, n_tiles = (g.nc + BN - 1) / BN;
  const int boxes = g.tiles_w * g.tiles_h * g.tiles_n;
  const int num_items = m_tiles * n_tiles * g.splits;
  const int ksteps = (g.pix + 15) >> 4;                      // MMAs (K = 16 pixels) per box

  // Rows of a stage buffer beyond the box's pixel count are never written by TMA; the last MMA of a box whose pixel
  // count is not a multiple of 16 reads up to 15 of them.  They are zeroed once here and stay zero.
  {
    uint4* p = reinterpret_cast<uint4*>(tiles);
    const int n16 = C::kStages * C::kStageBytes / 16;
    for (int i = threadIdx.x; i < n16; i += kWgThreads) p[i] = make_uint4(0, 0, 0, 0);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (threadIdx.x == 0) {
    for (int s = 0; s < C::kStages; ++s) {
      mbar_init(full_bar + s, 1);
      mbar_init(empty_bar + s, 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(tmem_full_bar + a, 1);
      mbar_init(tmem_empty_bar + a, 4);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&xmaps.m[0]) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&dymap) : "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"((uint32_t)C::kTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = *tmem_slot;
  tsp::wait_for_previous();

  if (warp == 0) {
    // ---------------- TMA producer ----------------
    if (lane == 0) {
      uint32_t it = 0;
      bool ok = true;
      const uint32_t tx = (uint32_t)((2 + BN / 64) * g.pix * 128);
      for (int item = blockIdx.x; item < num_items && ok; item += gridDim.x) {
        const int mt = item % m_tiles, nt = (item / m_tiles) % n_tiles, sp = item / (m_tiles * n_tiles);
        const int b_lo = (int)((int64_t)boxes * sp / g.splits), b_hi = (int)((int64_t)boxes * (sp + 1) / g.splits);
        int mb[2] = {2 * mt, 2 * mt + 1};
        if (mb[1] >= m_blocks) mb[1] = mb[0];                 // odd block count: the last tile's upper half is a copy
        for (int bx = b_lo; bx < b_hi; ++bx, ++it) {
          int w0, h0, n0;
          tile_origin(g, bx, w0, h0, n0);
          const int s = it % C::kStages;
          if (it % C::kGroup == 0) {
            const uint32_t grp = (it / C::kGroup) % C::kGroups, round = (it / C::kGroup) / C::kGroups;
            if (round > 0 && !mbar_wait_parked(empty_bar + grp, (round - 1) & 1, status, 1, g.wait_ns)) { ok = false; break; }
          }
          uint8_t* a_dst = tiles + s * C::kStageBytes;
          uint8_t* b_dst = a_dst + C::kABytes;
          mbar_expect_tx(full_bar + s, tx);
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int tap = mb[h] / kcb, cb = mb[h] % kcb;
            tma_load_4d(a_dst + h * C::kBox, &xmaps.m[g.tap_map[tap]], full_bar + s, cb * 64, w0 + g.tap_dw[tap],
                        h0 + g.tap_dh[tap], n0);
          }
#pragma unroll
          for (int j = 0; j < BN / 64; ++j)                    // channel blocks past nc read as zeros
            tma_load_4d(b_dst + j * C::kBox, &dymap, full_bar + s, nt * BN + j * 64, w0, h0, n0);
        }
      }
      tsp::let_next_start();
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer ----------------
    {
      const bool issuer = tc5::elect_one();
      auto arrived = [&](uint64_t* bar, uint32_t parity, int code) -> bool {      // the same for the warp
        return __all_sync(0xffffffffu, tc5::mbar_wait(bar, parity, status, code, g.wait_ns)) != 0;
      };
      constexpr uint32_t idesc = make_idesc(128, BN, true, true);
      const uint32_t tiles_addr = smem_u32(tiles);
      uint32_t it = 0, lt = 0;
      bool ok = true;
      for (int item = blockIdx.x; item < num_items && ok; item += gridDim.x, ++lt) {
        const int sp = item / (m_tiles * n_tiles);
        const int b_lo = (int)((int64_t)boxes * sp / g.splits), b_hi = (int)((int64_t)boxes * (sp + 1) / g.splits);
        const uint32_t acc = lt & 1, use = lt >> 1;
        if (use > 0) {
          ok = arrived(tmem_empty_bar + acc, (use - 1) & 1, 4);
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        }
        const uint32_t d_tmem = tmem_base + acc * BN;
        uint32_t accum = 0u;
        for (int bx = b_lo; bx < b_hi; ++bx, ++it) {
          const int s = it % C::kStages;
          const uint32_t round = it / C::kStages;
          ok = arrived(full_bar + s, round & 1, 2);
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t a_addr = tiles_addr + s * C::kStageBytes;
          const uint32_t a_dlo = desc_lo_mn_major(a_addr, C::kBox), b_dlo = desc_lo_mn_major(a_addr + C::kABytes, C::kBox);
          for (int ks = 0; ks < ksteps; ++ks) {                     // 16 pixels further on: +2048 bytes
            if (issuer) umma_bf16_lo(d_tmem, a_dlo + 128 * ks, b_dlo + 128 * ks, idesc, accum);
            accum = 1u;
          }
          if (issuer && it % C::kGroup == C::kGroup - 1) umma_commit(empty_bar + (it / C::kGroup) % C::kGroups);
        }
        if (issuer) umma_commit(tmem_full_bar + acc);
      }
    }
  } else {
    // ---------------- epilogue: add the partial tile into dW[co][(tap, ci)] ----------------
    const int quarter = warp & 3;
    uint32_t lt = 0;
    bool ok = true;
    for (int item = blockIdx.x; item < num_items && ok; item += gridDim.x, ++lt) {
      const int mt = item % m_tiles, nt = (item / m_tiles) % n_tiles, sp = item / (m_tiles * n_tiles);
      const int b_lo = (int)((int64_t)boxes * sp / g.splits), b_hi = (int)((int64_t)boxes * (sp + 1) / g.splits);
      const uint32_t acc = lt & 1, use = lt >> 1;
      ok = mbar_wait_warp(tmem_full_bar + acc, use & 1, status, 3, g.wait_ns, lane);
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const int m = mt * 128 + quarter * 32 + lane;             // index into the (tap, ci) axis
      // an empty pixel range leaves the accumulator unset, a wait that ran out may leave part of a sum in it
      const bool row_ok = m < m_blocks * 64 && b_hi > b_lo && *((volatile int*)status) == 0;
#pragma unroll 1
      for (int c0 = 0; c0 < BN; c0 += 32) {
        const int co0 = nt * BN + c0;
        if (co0 >= g.nc) break;
        uint32_t r[32];
        tmem_ld_32x32_issue(tmem_base + ((uint32_t)(quarter * 32) << 16) + acc * BN + (uint32_t)c0, r);
        tmem_ld_wait();
        if (row_ok) {
          float* dst = dw + (int64_t)co0 * g.ldw + m;
#pragma unroll
          for (int j = 0; j < 32; ++j)
            if (co0 + j < g.nc) atomicAdd(dst + (int64_t)j * g.ldw, __uint_as_float(r[j]));
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(tmem_empty_bar + acc);
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)C::kTmemCols)
                 : "memory");
  }
}

// ---------------------------------------------------------------------------------------------------------------
// weight gradient of a 3x3 stride-1 convolution of 64 to 64 channels with the bordered pixel box resident
// ---------------------------------------------------------------------------------------------------------------
// conv_wgrad_kernel fetches a shifted box per tap (15 boxes of 16 KB per 128 pixels, bound by L2).  Here a tile's bordered
// box of x and its box of dY come once, both enumerated in the bordered pitch (dY's border columns are zero-filled by TMA
// and cancel what x holds there), and the operand of tap (kh, kw) is the resident box read from row kh * pitch + kw on, as
// in conv_halo_kernel.  M = two taps (their 64-channel blocks LBO apart: the distance of the two shifts), N = co, K = the
// box's rows; the nine taps' accumulators, five of 128 x 64, stay in tensor memory over all tiles of a CTA.  An infinite or
// NaN x in an image's first or last column or row meets those zeros too, in taps that do not pair it with a dY: sums that
// come out infinite or NaN are formed again from the definition (add_wgrad_exact), so that they are so where they should be.
// 256 images of 56 x 56, B200: 137 us with conv_wgrad_kernel, 79 with this one (67 once the products were issued by a converged warp).
struct WgHaloCfg {
  static constexpr int kXBytes = 384 * 128;                     // bordered box: up to 256 + 2 pitches + 2 rows
  static constexpr int kDyBytes = 256 * 128;
  static constexpr int kStageBytes = kXBytes + kDyBytes;
  static constexpr int kStages = 2;
  static constexpr int kPairs = 5;
  static constexpr int kTmemCols = 512;
  static constexpr int kSmemBytes = kStages * kStageBytes + 1024 + 256;
};
// The share of a CTA's tiles in dW[co0 .. co0 + 31][tap][ci], one (tap, ci) per thread, as the sum over its pixels of dY and
// the zero-padded x.
__device__ __noinline__ void add_wgrad_exact(const Geom& g, const __nv_bfloat16* __restrict__ x,
                                             const __nv_bfloat16* __restrict__ dy, int t_begin, int t_end, int tap, int ci,
                                             int co0, float* __restrict__ dw) {
  float acc[32];
#pragma unroll
  for (int j = 0; j < 32; ++j) acc[j] = 0.f;
  for (int t = t_begin; t < t_end; ++t) {
    int w0, h0, n0;
    tile_origin(g, t, w0, h0, n0);
    for (int h = h0; h < min(h0 + g.box_h, g.out_h); ++h)
      for (int w = 0; w < g.out_w; ++w) {
        const int xh = h + tap / 3 - 1, xw = w + tap % 3 - 1;
        const bool inside = xh >= 0 && xh < g.out_h && xw >= 0 && xw < g.out_w;
        const float xv = inside ? __bfloat162float(x[(((int64_t)n0 * g.out_h + xh) * g.out_w + xw) * 64 + ci]) : 0.f;
        const __nv_bfloat16* row = dy + (((int64_t)n0 * g.out_h + h) * g.out_w + w) * 64 + co0;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          float v[8];
          tsp::ld8(row, q * 8, v);
#pragma unroll
          for (int e = 0; e < 8; ++e) acc[q * 8 + e] = fmaf(xv, v[e], acc[q * 8 + e]);
        }
      }
  }
#pragma unroll
  for (int j = 0; j < 32; ++j) atomicAdd(dw + (int64_t)(co0 + j) * 576 + tap * 64 + ci, acc[j]);
}
__device__ __forceinline__ int first_tap(int pair) { return pair < 4 ? 2 * pair : 7; }      // the last pair repeats tap 7

__global__ void __launch_bounds__(kWgThreads, 1)
conv_wgrad_halo_kernel(const __grid_constant__ CUtensorMap xmap, const __grid_constant__ CUtensorMap dymap,
                       const __grid_constant__ Geom g, const __nv_bfloat16* __restrict__ x,
                       const __nv_bfloat16* __restrict__ dy, float* __restrict__ dw, int* __restrict__ status) {
  extern __shared__ uint8_t smem_raw[];
  using C = WgHaloCfg;
  uint8_t* tiles = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint64_t* bars = (uint64_t*)(tiles + C::kStages * C::kStageBytes);
  uint64_t* full_bar = bars;
  uint64_t* empty_bar = bars + C::kStages;
  uint64_t* done_bar = bars + 2 * C::kStages;
  uint32_t* tmem_slot = (uint32_t*)(bars + 2 * C::kStages + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int num_tiles = g.tiles_w * g.tiles_h * g.tiles_n;
  const int t_begin = tile_begin(num_tiles, blockIdx.x), t_end = tile_begin(num_tiles, blockIdx.x + 1);
  const int ksteps = (g.pix + 15) >> 4;

  // Rows past the boxes are never written by TMA but are read: by the last 16 rows of dY's K loop, where zeros have to meet
  // finite values, and by shifted starts in x.  Zeroed once, they stay zero.
  {
    uint4* p = reinterpret_cast<uint4*>(tiles);
    for (int i = threadIdx.x; i < C::kStages * C::kStageBytes / 16; i += kWgThreads) p[i] = make_uint4(0, 0, 0, 0);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (threadIdx.x == 0) {
    for (int s = 0; s < C::kStages; ++s) { mbar_init(full_bar + s, 1); mbar_init(empty_bar + s, 1); }
    mbar_init(done_bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&xmap) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&dymap) : "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"((uint32_t)C::kTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = *tmem_slot;
  tsp::wait_for_previous();
  x = tsp::written(x); dy = tsp::written(dy);

  if (warp == 0) {
    // ---------------- TMA producer ----------------
    if (lane == 0) {
      const uint32_t tx = (uint32_t)((g.halo_rows + g.pix) * 128);
      for (int t = t_begin; t < t_end; ++t) {
        const int it = t - t_begin, s = it % C::kStages;
        const uint32_t round = (uint32_t)it / C::kStages;
        if (round > 0 && !mbar_wait_parked(empty_bar + s, (round - 1) & 1, status, 1, g.wait_ns)) break;
        int w0, h0, n0;
        tile_origin(g, t, w0, h0, n0);
        uint8_t* dst = tiles + s * C::kStageBytes;
        mbar_expect_tx(full_bar + s, tx);
        tma_load_4d(dst, &xmap, full_bar + s, 0, w0 - 1, h0 - 1, n0);
        tma_load_4d(dst + C::kXBytes, &dymap, full_bar + s, 0, w0, h0, n0);
      }
      tsp::let_next_start();
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer ----------------
    {
      const bool issuer = tc5::elect_one();
      auto arrived = [&](uint64_t* bar, uint32_t parity, int code) -> bool {      // the same for the warp
        return __all_sync(0xffffffffu, tc5::mbar_wait(bar, parity, status, code, g.wait_ns)) != 0;
      };
      constexpr uint32_t idesc = make_idesc(128, 64, true, true);
      const uint32_t tiles_addr = smem_u32(tiles);
      uint32_t accum = 0u;
      for (int t = t_begin; t < t_end; ++t) {
        const int it = t - t_begin, s = it % C::kStages;
        if (!arrived(full_bar + s, ((uint32_t)it / C::kStages) & 1, 2)) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t x_addr = tiles_addr + s * C::kStageBytes;
        const uint32_t b_lo = desc_lo_mn_major(x_addr + C::kXBytes, 8192);
        uint32_t a_lo[C::kPairs];
#pragma unroll
        for (int a = 0; a < C::kPairs; ++a) {
          const int o0 = g.tap_off[first_tap(a)], o1 = g.tap_off[first_tap(a) + 1];
          a_lo[a] = desc_lo_mn_major(x_addr + o0 * 128, (uint32_t)(o1 - o0) * 128u);
        }
        for (int ks = 0; ks < ksteps; ++ks) {                     // 16 rows further on: +2048 bytes
#pragma unroll
          for (int a = 0; a < C::kPairs; ++a)
            if (issuer) umma_bf16_lo(tmem_base + a * 64, a_lo[a] + 128 * ks, b_lo + 128 * ks, idesc, accum);
          accum = 1u;
        }
        if (issuer) umma_commit(empty_bar + s);
      }
      if (issuer) umma_commit(done_bar);
    }
  } else if (t_begin < t_end) {
    // ---------------- epilogue: add the accumulators into dW[co][(tap, ci)] ----------------
    const int quarter = warp & 3;
    if (mbar_wait_warp(done_bar, 0, status, 3, g.wait_ns, lane) && *((volatile int*)status) == 0) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const int m = quarter * 32 + lane;
#pragma unroll 1
      for (int a = 0; a < C::kPairs; ++a) {
        if (a == C::kPairs - 1 && quarter < 2) continue;
        const int tap = first_tap(a) + (m >> 6), ci = m & 63;
        float* dst = dw + tap * 64 + ci;
#pragma unroll 1
        for (int c0 = 0; c0 < 64; c0 += 32) {
          uint32_t r[32];
          tmem_ld_32x32_issue(tmem_base + ((uint32_t)(quarter * 32) << 16) + a * 64 + c0, r);
          tmem_ld_wait();
          bool finite = true;
#pragma unroll
          for (int j = 0; j < 32; ++j) finite = finite && (r[j] & 0x7f800000u) != 0x7f800000u;
          if (finite) {
#pragma unroll
            for (int j = 0; j < 32; ++j) atomicAdd(dst + (int64_t)(c0 + j) * 576, __uint_as_float(r[j]));
          } else {
            add_wgrad_exact(g, x, dy, t_begin, t_end, tap, ci, c0, dw);
          }
          __syncwarp();
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)C::kTmemCols)
                 : "memory");
  }
}

// One barrier that nothing ever completes, waited on with the same bounded wait the kernels above use: the wait gives
// up after `limit_ns`, leaves `code` in *status and the kernel returns normally.
__global__ void bounded_wait_probe_kernel(unsigned long long limit_ns, int code, int* status) {
  __shared__ uint64_t bar;
  if (threadIdx.x == 0) {
    mbar_init(&bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    mbar_wait(&bar, 0, status, code, limit_ns);
  }
}

// ---------------------------------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------------------------------
unsigned long long g_wait_ns = 2000000000ull;     // give-up time of the kernels' mbarrier waits (2 s)

}  // namespace
extern int g_tsp_sm_reserve;          // defined in peer.cu
namespace {

int sm_count() {
  static int n_sm[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  dev &= 63;
  if (n_sm[dev] == 0) {
    cudaDeviceGetAttribute(&n_sm[dev], cudaDevAttrMultiProcessorCount, dev);
    if (n_sm[dev] <= 0) n_sm[dev] = 148;
  }
  const int n = n_sm[dev] - g_tsp_sm_reserve;       // SMs left to communication kernels stay free
  return n > 8 ? n : 8;
}

// Pixel box for a w x h x n grid: at most max_pix pixels, as few tiles as possible, tiles of equal size where it
// divides.
void choose_box(int w, int h, int n, int max_pix, int& bw, int& bh, int& bn) {
  bw = w < max_pix ? w : max_pix;
  const int hmax = max_pix / bw;
  bh = 1;
  if (hmax > 1) {
    const int th = (h + hmax - 1) / hmax;           // tiles along h
    bh = (h + th - 1) / th;
  }
  const int nmax = max_pix / (bw * bh);
  bn = 1;
  if (nmax > 1 && bh >= h) {
    const int tn = (n + nmax - 1) / nmax;
    bn = (n + tn - 1) / tn;
  }
}

// Tensor map of a dense channels-last view: base + (c, w, h, n) with pitches pw / ph / pn ELEMENTS, box as given.
bool act_map(CUtensorMap* map, const void* base, int c, int w, int h, int n, int64_t pw, int64_t ph, int64_t pn, int bw,
             int bh, int bn) {
  const uint64_t dims[4] = {(uint64_t)c, (uint64_t)w, (uint64_t)h, (uint64_t)n};
  const uint64_t strides[4] = {2, (uint64_t)pw * 2, (uint64_t)ph * 2, (uint64_t)pn * 2};
  const uint32_t box[4] = {64, (uint32_t)bw, (uint32_t)bh, (uint32_t)bn};
  return make_bf16_map(map, base, 4, dims, strides, box);
}

// A convolution problem seen from its OUTPUT pixel grid: where the shifted input boxes come from.
struct Plan {
  Geom g;
  ActMaps maps;
  bool ok;
};

// Shifted-input side of the forward product (and of the weight gradient): input x [n, h, w, cin], kernel k, stride s.
// `flat` = 1x1 stride 1: all pixels as one row of n*h*w.
Plan plan_input(const void* x, int n, int h, int w, int cin, int k, int s, int max_pix = 128) {
  Plan p = {};
  Geom& g = p.g;
  const int pad = (k - 1) / 2;
  const bool flat = k == 1 && s == 1;
  const int ho = (h + 2 * pad - k) / s + 1, wo = (w + 2 * pad - k) / s + 1;
  if (flat) {
    g.out_w = n * h * w; g.out_h = 1; g.out_n = 1;
  } else {
    g.out_w = wo; g.out_h = ho; g.out_n = n;
  }
  choose_box(g.out_w, g.out_h, g.out_n, max_pix, g.box_w, g.box_h, g.box_n);
  g.tiles_w = (g.out_w + g.box_w - 1) / g.box_w;
  g.tiles_h = (g.out_h + g.box_h - 1) / g.box_h;
  g.tiles_n = (g.out_n + g.box_n - 1) / g.box_n;
  g.row_pitch = g.box_w;
  g.pix = g.box_w * g.box_h * g.box_n;
  g.wait_ns = g_wait_ns;
  g.n_taps = k * k;
  g.kc = cin;
  p.ok = true;
  if (flat) {
    p.ok = act_map(&p.maps.m[0], x, cin, g.out_w, 1, 1, cin, (int64_t)cin * g.out_w, (int64_t)cin * g.out_w, g.box_w, 1, 1);
    for (int i = 1; i < 4; ++i) p.maps.m[i] = p.maps.m[0];
    g.tap_dw[0] = g.tap_dh[0] = g.tap_map[0] = g.tap_col[0] = 0;
    return p;
  }
  if (s == 1) {
    p.ok = act_map(&p.maps.m[0], x, cin, w, h, n, cin, (int64_t)w * cin, (int64_t)h * w * cin, g.box_w, g.box_h, g.box_n);
    for (int i = 1; i < 4; ++i) p.maps.m[i] = p.maps.m[0];
  } else {
    // one dense view per (row parity, column parity): x[n, 2a + ph, 2b + pw, :]
    for (int ph = 0; ph < 2 && p.ok; ++ph)
      for (int pw = 0; pw < 2 && p.ok; ++pw) {
        const __nv_bfloat16* base = (const __nv_bfloat16*)x + ((int64_t)ph * w + pw) * cin;
        p.ok = act_map(&p.maps.m[ph * 2 + pw], base, cin, w / 2, h / 2, n, 2 * (int64_t)cin, 2 * (int64_t)w * cin,
                       (int64_t)h * w * cin, g.box_w, g.box_h, g.box_n);
      }
  }
  for (int kh = 0; kh < k; ++kh)
    for (int kw = 0; kw < k; ++kw) {
      const int t = kh * k + kw;
      const int dh = kh - pad, dw_ = kw - pad;            // input row = s * ho + dh
      if (s == 1) {
        g.tap_dh[t] = dh; g.tap_dw[t] = dw_; g.tap_map[t] = 0;
      } else {
        const int ph = dh & 1, pw = dw_ & 1;              // parity of the input row / column (two's complement: -1 -> 1)
        g.tap_dh[t] = (dh - ph) / 2; g.tap_dw[t] = (dw_ - pw) / 2; g.tap_map[t] = ph * 2 + pw;
      }
      g.tap_col[t] = t * cin;
    }
  return p;
}

template <int BN, bool B_MN, bool STATS, int ADD, int GROUPS = 2>
int launch_fwd_kernel(const Plan& p, const CUtensorMap& wmap, const CUtensorMap& omap, const CUtensorMap& addmap, const Geom& g,
                      void* out, const void* addend, float* col_sums, int* status, cudaStream_t stream) {
  auto kern = conv_fwd_kernel<BN, B_MN, STATS, ADD, GROUPS>;
  using C = FwdCfg<BN, ADD, GROUPS>;
  static bool attr_set[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  dev &= 63;
  if (!attr_set[dev]) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmemBytes);
    if (e != cudaSuccess) return (int)e;
    attr_set[dev] = true;
  }
  const int num_tiles = g.tiles_w * g.tiles_h * g.tiles_n * ((g.nc + BN - 1) / BN);
  const int n_sm = sm_count();
  const int grid = num_tiles < n_sm ? num_tiles : n_sm;
  tsp::launch_early(kern, grid, C::kThreads, C::kSmemBytes, stream, p.maps, wmap, omap, addmap, g, (__nv_bfloat16*)out,
                    (const __nv_bfloat16*)addend, col_sums, status);
  return TSP_LAUNCH_CHECK();
}

template <int BN, bool B_MN, bool STATS, bool ADD>
int launch_fwd(const Plan& p, const CUtensorMap& wmap, void* out, const void* addend, float* col_sums, int* status,
               cudaStream_t stream) {
  Geom g = p.g;
  // flat pixel grid (1x1 stride 1, dense output rows): [pixels, nc] matrix written in 32-row x 64-channel TMA stores
  CUtensorMap omap = wmap, addmap = wmap;
  g.tma_store = 0;
  g.n_fastest = STATS ? 0 : 1;
  set_divisors(g, (g.nc + BN - 1) / BN);
  if (g.out_h == 1 && g.out_n == 1 && g.out_sw * 8 == g.nc && g.box_w == 128) {
    const uint64_t dims[2] = {(uint64_t)g.nc, (uint64_t)g.out_w};
    const uint64_t strides[2] = {2, (uint64_t)g.nc * 2};
    const uint32_t box[2] = {64, 32};
    if (make_bf16_map(&omap, out, 2, dims, strides, box)) g.tma_store = 1;
    if constexpr (ADD) {
      if (g.tma_store != 0 && make_bf16_map(&addmap, addend, 2, dims, strides, box))
        return launch_fwd_kernel<BN, B_MN, STATS, 2>(p, wmap, omap, addmap, g, out, addend, col_sums, status, stream);
    }
  }
  // Statistics after a short contraction: the epilogue is what a tile waits for, and it has too few warps to fill their waits.
  // B200, 8 warps against 16 (and one operand stage less): 256 images of 56 x 56, 64 -> 256 110 us and 101, 64 images of
  // 28 x 28, 128 -> 512 21.2 and 20.0, of 14 x 14, 256 -> 1024 16.4 and 15.3; 512 -> 128 at 28 x 28 16.0 and 17.1.
  if constexpr (STATS) {
    if (g.n_taps * g.kc < 512)
      return launch_fwd_kernel<BN, B_MN, STATS, ADD ? 1 : 0, 4>(p, wmap, omap, addmap, g, out, addend, col_sums, status, stream);
  }
  return launch_fwd_kernel<BN, B_MN, STATS, ADD ? 1 : 0>(p, wmap, omap, addmap, g, out, addend, col_sums, status, stream);
}

template <bool B_MN, bool STATS, bool ADD = false>
int dispatch_fwd(int bn, const Plan& p, const CUtensorMap& wmap, void* out, const void* addend, float* col_sums,
                 int* status, cudaStream_t stream) {
  if (bn == 256) return launch_fwd<256, B_MN, STATS, ADD>(p, wmap, out, addend, col_sums, status, stream);
  if (bn == 128) return launch_fwd<128, B_MN, STATS, ADD>(p, wmap, out, addend, col_sums, status, stream);
  return launch_fwd<64, B_MN, STATS, ADD>(p, wmap, out, addend, col_sums, status, stream);
}

// 3x3 stride-1 walk over an image grid with the bordered box kept in shared memory (conv_halo_kernel): applies when
// a bordered row fits (w <= 61) and the image is large enough that one box per image does not waste the tile.
bool halo_applies(int k, int s, int w, int h) {
  static int enabled = -1;
  if (enabled < 0) {
    const char* e = getenv("TSP_CONV_HALO");
    enabled = (e != nullptr && e[0] == '0') ? 0 : 1;
  }
  return enabled && k == 3 && s == 1 && w <= 61 && h * (w + 2) > 64;
}

// Geometry of the halo kernel over src[n, h, w, c] (the forward's input, or dy for the data gradient).
bool plan_halo(Geom& g, CUtensorMap* amap, const void* src, int n, int h, int w, int c) {
  g = Geom{};
  const int pitch = w + 2, hmax = 256 / pitch;        // up to 256 accumulator rows (two accumulators) per tile
  const int th = (h + hmax - 1) / hmax;
  g.out_w = w; g.out_h = h; g.out_n = n;
  g.box_w = w; g.box_h = (h + th - 1) / th; g.box_n = 1;
  g.tiles_w = 1; g.tiles_h = th; g.tiles_n = n;
  g.row_pitch = pitch;
  g.pix = pitch * g.box_h;
  g.halo_rows = pitch * (g.box_h + 2);
  g.n_taps = 9;
  g.kc = c;
  g.rows_per_seg = 1 << 30;
  g.wait_ns = g_wait_ns;
  return act_map(amap, src, c, w, h, n, c, (int64_t)w * c, (int64_t)h * w * c, pitch, g.box_h + 2, 1);
}

template <int BN, bool B_MN, bool STATS, bool ADD>
int launch_halo(Geom& g, const CUtensorMap& amap, const CUtensorMap& wmap, void* out, const void* addend, float* col_sums,
                int* status, cudaStream_t stream) {
  g.n_fastest = STATS ? 0 : 1;
  set_divisors(g, (g.nc + BN - 1) / BN);
  auto kern = conv_halo_kernel<BN, B_MN, STATS, ADD>;
  static bool attr_set[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  dev &= 63;
  if (!attr_set[dev]) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, HaloCfg<BN>::kSmemBytes);
    if (e != cudaSuccess) return (int)e;
    attr_set[dev] = true;
  }
  const int num_tiles = g.tiles_w * g.tiles_h * g.tiles_n * ((g.nc + BN - 1) / BN);
  const int n_sm = sm_count();
  const int grid = num_tiles < n_sm ? num_tiles : n_sm;
  tsp::launch_early(kern, grid, kThreads, HaloCfg<BN>::kSmemBytes, stream, amap, wmap, g, (__nv_bfloat16*)out,
                    (const __nv_bfloat16*)addend, col_sums, status);
  return TSP_LAUNCH_CHECK();
}

template <bool B_MN, bool STATS, bool ADD = false>
int dispatch_halo(int bn, Geom& g, const CUtensorMap& amap, const CUtensorMap& wmap, void* out, const void* addend,
                  float* col_sums, int* status, cudaStream_t stream) {
  g.b_resident = (bn == 64 && g.kc == 64 && g.nc == 64) ? 1 : 0;      // 9 weight tiles = the 9 ring slots
  if (bn == 256) return launch_halo<256, B_MN, STATS, ADD>(g, amap, wmap, out, addend, col_sums, status, stream);
  if (bn == 128) return launch_halo<128, B_MN, STATS, ADD>(g, amap, wmap, out, addend, col_sums, status, stream);
  return launch_halo<64, B_MN, STATS, ADD>(g, amap, wmap, out, addend, col_sums, status, stream);
}

// Output channels per tile, given the number of pixel tiles: the most that divide nc, halved while all tiles of the narrower
// width still run at once.  Image grids of the
// last two stages of a ResNet-50 over 64 images, B200: 3 x 3 at 14 x 14 34 us at 256 channels on 64 SMs, 25.7 at 128 on 128; at
// 7 x 7 35.6 and 28.  More tiles than SMs cost a second round: 1024 -> 256 at 14 x 14 (98 tiles) stays at 256.
int pick_bn(int nc, int64_t tiles_m) {
  int bn = nc % 256 == 0 ? 256 : (nc % 128 == 0 ? 128 : 64);
  while (bn > 64 && tiles_m * (nc / (bn / 2)) <= sm_count()) bn /= 2;
  return bn;
}
int64_t pixel_tiles(const Geom& g) { return (int64_t)g.tiles_w * g.tiles_h * g.tiles_n; }

template <int BN>
int launch_wgrad(const Plan& p, const CUtensorMap& dymap, float* dw, int* status, cudaStream_t stream) {
  auto kern = conv_wgrad_kernel<BN>;
  static bool attr_set[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  dev &= 63;
  if (!attr_set[dev]) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, WgCfg<BN>::kSmemBytes);
    if (e != cudaSuccess) return (int)e;
    attr_set[dev] = true;
  }
  Geom g = p.g;
  set_divisors(g, 1);
  const int m_tiles = (g.n_taps * (g.kc / 64) + 1) / 2, n_tiles = (g.nc + BN - 1) / BN;
  const int items = m_tiles * n_tiles * g.splits;
  const int n_sm = sm_count();
  const int grid = items < n_sm ? items : n_sm;
  tsp::launch_early(kern, grid, kWgThreads, WgCfg<BN>::kSmemBytes, stream, p.maps, dymap, g, dw, status);
  return TSP_LAUNCH_CHECK();
}

int launch_wgrad_halo(const void* x, const void* dy, float* dw, int n, int h, int w, int* status, cudaStream_t stream) {
  Geom g;
  CUtensorMap xmap, dymap;
  if (!plan_halo(g, &xmap, x, n, h, w, 64) ||
      !act_map(&dymap, dy, 64, w, h, n, 64, (int64_t)w * 64, (int64_t)h * w * 64, g.row_pitch, g.box_h, 1))
    return -6;
  for (int t = 0; t < 9; ++t) g.tap_off[t] = (t / 3) * g.row_pitch + t % 3;
  set_divisors(g, 1);
  auto kern = conv_wgrad_halo_kernel;
  static bool attr_set[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  dev &= 63;
  if (!attr_set[dev]) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, WgHaloCfg::kSmemBytes);
    if (e != cudaSuccess) return (int)e;
    attr_set[dev] = true;
  }
  const int num_tiles = g.tiles_w * g.tiles_h * g.tiles_n;
  const int n_sm = sm_count();
  tsp::launch_early(kern, num_tiles < n_sm ? num_tiles : n_sm, kWgThreads, WgHaloCfg::kSmemBytes, stream, xmap, dymap, g,
                    (const __nv_bfloat16*)x, (const __nv_bfloat16*)dy, dw, status);
  return TSP_LAUNCH_CHECK();
}

bool shape_ok(int n, int h, int w, int cin, int cout, int k, int s) {
  if (n <= 0 || h <= 0 || w <= 0) return false;
  if (cin % 64 || cout % 64 || cin <= 0 || cout <= 0) return false;
  if (!(k == 1 || k == 3) || !(s == 1 || s == 2)) return false;
  if (s == 2 && ((h | w) & 1)) return false;
  return true;
}

}  // namespace

extern "C" {

// Give-up time (milliseconds, default 2000) of every mbarrier wait in the kernels of this file launched afterwards.
void tsp_conv_set_wait_limit_ms(int ms) { g_wait_ns = (unsigned long long)(ms > 0 ? ms : 1) * 1000000ull; }

// Failure-detection self-test: runs the kernels' bounded mbarrier wait on a barrier that is never completed.  After
// about `limit_ms` milliseconds the wait gives up, *status (one zeroed int in device memory) becomes `code`, and the
// kernel ends normally: nothing traps, the context stays usable.
int tsp_bounded_wait_probe(int limit_ms, int code, int* status, cudaStream_t stream) {
  if (limit_ms < 1 || limit_ms > 2000) return -3;
  bounded_wait_probe_kernel<<<1, 32, 0, stream>>>((unsigned long long)limit_ms * 1000000ull, code, status);
  return TSP_LAUNCH_CHECK();
}

// y[n, ho, wo, cout] = conv(x[n, h, w, cin], wgt[cout][k][k][cin]), stride s, padding (k - 1) / 2; all bf16,
// channels-last, 16-byte aligned, cin and cout multiples of 64.  col_sums (optional, zeroed by the caller):
// [segs][2 * cout] fp32 receives per-channel sum and sum of squares of y over each of `segs` equal groups of
// consecutive images (n divisible by segs; for a 1x1 stride-1 convolution of several groups the pixels per group must be a
// multiple of 128).  `status`: one zeroed int in device memory; non-zero afterwards = a bounded wait ran out, y is not valid.
int tsp_conv_fprop(const void* x, const void* wgt, void* y, float* col_sums, int segs, int n, int h, int w, int cin,
                   int cout, int k, int s, int* status, cudaStream_t stream) {
  if (!shape_ok(n, h, w, cin, cout, k, s)) return -3;
  if (((uintptr_t)x | (uintptr_t)wgt | (uintptr_t)y) & 15) return -2;
  const int pad = (k - 1) / 2, ho = (h + 2 * pad - k) / s + 1, wo = (w + 2 * pad - k) / s + 1;
  if ((int64_t)n * ho * wo * cout / 8 >= (int64_t)1 << 31) return -3;
  if (halo_applies(k, s, w, h)) {
    Geom g;
    CUtensorMap amap, wmap;
    if (!plan_halo(g, &amap, x, n, h, w, cin)) return -6;
    g.nc = cout;
    for (int t = 0; t < 9; ++t) { g.tap_off[t] = (t / 3) * g.row_pitch + t % 3; g.tap_col[t] = t * cin; }
    g.out_sw = cout / 8; g.out_sh = w * (cout / 8); g.out_sn = h * w * (cout / 8);
    if (col_sums != nullptr) {
      if (segs < 1 || n % segs) return -3;
      g.rows_per_seg = (int)((int64_t)n * h * w / segs);
    }
    const int bn = pick_bn(cout, pixel_tiles(g));
    const uint64_t dims[2] = {(uint64_t)9 * cin, (uint64_t)cout};
    const uint64_t strides[2] = {2, (uint64_t)9 * cin * 2};
    const uint32_t box[2] = {64, (uint32_t)bn};
    if (!make_bf16_map(&wmap, wgt, 2, dims, strides, box)) return -6;
    if (col_sums != nullptr) return dispatch_halo<false, true>(bn, g, amap, wmap, y, nullptr, col_sums, status, stream);
    return dispatch_halo<false, false>(bn, g, amap, wmap, y, nullptr, nullptr, status, stream);
  }
  Plan p = plan_input(x, n, h, w, cin, k, s);
  if (!p.ok) return -6;
  Geom& g = p.g;
  g.nc = cout;
  const bool flat = k == 1 && s == 1;
  g.out_sw = cout / 8;
  g.out_sh = flat ? 0 : wo * (cout / 8);
  g.out_sn = flat ? 0 : ho * wo * (cout / 8);
  g.rows_per_seg = 1 << 30;
  if (col_sums != nullptr) {
    if (segs < 1 || n % segs) return -3;
    const int64_t rows = (int64_t)n * ho * wo / segs;
    if (flat && segs > 1 && rows % 128) return -3;
    if (!flat && g.box_n > 1 && (n / segs) % g.box_n) return -3;
    g.rows_per_seg = (int)rows;
  }
  const int bn = pick_bn(cout, pixel_tiles(g));
  CUtensorMap wmap;
  const uint64_t dims[2] = {(uint64_t)k * k * cin, (uint64_t)cout};
  const uint64_t strides[2] = {2, (uint64_t)k * k * cin * 2};
  const uint32_t box[2] = {64, (uint32_t)bn};
  if (!make_bf16_map(&wmap, wgt, 2, dims, strides, box)) return -6;
  if (col_sums != nullptr) return dispatch_fwd<false, true>(bn, p, wmap, y, nullptr, col_sums, status, stream);
  return dispatch_fwd<false, false>(bn, p, wmap, y, nullptr, nullptr, status, stream);
}

// dx[n, h, w, cin] = gradient of tsp_conv_fprop's input given dy[n, ho, wo, cout] and the same weights
// wgt[cout][k][k][cin] (read in place through MN-major operand tiles).  Every element of dx is written.  `addend`
// (optional, dx's shape and layout; not for a 1x1 kernel of stride 2): added to the rounded result, the gradient that
// reaches the input on another way (a residual connection).  The gradient of
// [256, 56, 56, 256], B200: 157 us with it, 91 and 172 for the product and a separate addition.
int tsp_conv_dgrad(const void* dy, const void* wgt, const void* addend, void* dx, int n, int h, int w, int cin, int cout,
                   int k, int s, int* status, cudaStream_t stream) {
  if (!shape_ok(n, h, w, cin, cout, k, s)) return -3;
  if (((uintptr_t)dy | (uintptr_t)wgt | (uintptr_t)dx | (uintptr_t)addend) & 15) return -2;
  if (addend != nullptr && k == 1 && s == 2) return -3;         // three of its four parity classes never reach a kernel
  const int pad = (k - 1) / 2, ho = (h + 2 * pad - k) / s + 1, wo = (w + 2 * pad - k) / s + 1;
  if ((int64_t)n * h * w * cin / 8 >= (int64_t)1 << 31) return -3;
  CUtensorMap wmap;                       // rows = co (contraction), columns = (tap, ci): boxes of 64 x 64
  const uint64_t dims[2] = {(uint64_t)k * k * cin, (uint64_t)cout};
  const uint64_t strides[2] = {2, (uint64_t)k * k * cin * 2};
  const uint32_t box[2] = {64, 64};
  if (!make_bf16_map(&wmap, wgt, 2, dims, strides, box)) return -6;
  if (halo_applies(k, s, wo, ho)) {
    Geom g;
    CUtensorMap amap;
    if (!plan_halo(g, &amap, dy, n, ho, wo, cout)) return -6;
    g.nc = cin;
    const int bn = pick_bn(cin, pixel_tiles(g));
    for (int t = 0; t < 9; ++t) {              // dx[p] takes tap (kh, kw) from dy[p + (1 - kh, 1 - kw)]
      g.tap_off[t] = (2 - t / 3) * g.row_pitch + (2 - t % 3);
      g.tap_col[t] = t * cin;
    }
    g.out_sw = cin / 8; g.out_sh = w * (cin / 8); g.out_sn = h * w * (cin / 8);
    if (addend != nullptr) return dispatch_halo<true, false, true>(bn, g, amap, wmap, dx, addend, nullptr, status, stream);
    return dispatch_halo<true, false>(bn, g, amap, wmap, dx, nullptr, nullptr, status, stream);
  }
  if (s == 1) {
    // dx[p] = sum_tap dy[p + (pad - kh, pad - kw)] w[:, kh, kw, :]: the forward kernel over dy with mirrored offsets
    Plan p = plan_input(dy, n, ho, wo, cout, k, 1);
    if (!p.ok) return -6;
    Geom& g = p.g;
    g.nc = cin;
    const int bn = pick_bn(cin, pixel_tiles(g));
    for (int kh = 0; kh < k; ++kh)
      for (int kw = 0; kw < k; ++kw) {
        const int t = kh * k + kw;
        g.tap_dh[t] = pad - kh; g.tap_dw[t] = pad - kw; g.tap_map[t] = 0; g.tap_col[t] = t * cin;
      }
    const bool flat = k == 1;
    g.out_sw = cin / 8;
    g.out_sh = flat ? 0 : w * (cin / 8);
    g.out_sn = flat ? 0 : h * w * (cin / 8);
    g.rows_per_seg = 1 << 30;
    if (addend != nullptr) return dispatch_fwd<true, false, true>(bn, p, wmap, dx, addend, nullptr, status, stream);
    return dispatch_fwd<true, false>(bn, p, wmap, dx, nullptr, nullptr, status, stream);
  }
  // stride 2: dx[n, 2a + ph, 2b + pw] gets the taps with kh = ph + pad (mod 2), from dy[a + (ph + pad - kh) / 2, ...].
  // One launch per parity class over the (h / 2) x (w / 2) grid of that class; a class no tap reaches is zero
  // (1x1 stride 2: only the even / even class receives anything).
  if (k == 1) {
    cudaError_t e = cudaMemsetAsync(dx, 0, (size_t)n * h * w * cin * 2, stream);
    if (e != cudaSuccess) return (int)e;
  }
  for (int ph = 0; ph < 2; ++ph)
    for (int pw = 0; pw < 2; ++pw) {
      Plan p = plan_input(dy, n, ho, wo, cout, 3, 1);       // geometry of a dense walk over dy's grid (taps set below)
      if (!p.ok) return -6;
      Geom& g = p.g;
      g.nc = cin;
      const int bn = pick_bn(cin, pixel_tiles(g));
      int nt = 0;
      for (int kh = 0; kh < k; ++kh)
        for (int kw = 0; kw < k; ++kw) {
          if (((ph + pad - kh) & 1) || ((pw + pad - kw) & 1)) continue;
          g.tap_dh[nt] = (ph + pad - kh) / 2; g.tap_dw[nt] = (pw + pad - kw) / 2; g.tap_map[nt] = 0;
          g.tap_col[nt] = (kh * k + kw) * cin;
          ++nt;
        }
      g.n_taps = nt;
      __nv_bfloat16* base = (__nv_bfloat16*)dx + ((int64_t)ph * w + pw) * cin;
      if (nt == 0) continue;                                 // zero, written by the memset above
      g.out_sw = 2 * cin / 8;
      g.out_sh = 2 * w * (cin / 8);
      g.out_sn = h * w * (cin / 8);
      g.rows_per_seg = 1 << 30;
      const __nv_bfloat16* add = addend == nullptr ? nullptr : (const __nv_bfloat16*)addend + (base - (__nv_bfloat16*)dx);
      const int rc = add != nullptr ? dispatch_fwd<true, false, true>(bn, p, wmap, base, add, nullptr, status, stream)
                                    : dispatch_fwd<true, false>(bn, p, wmap, base, nullptr, nullptr, status, stream);
      if (rc != 0) return rc;
    }
  return 0;
}

// dw[cout][k][k][cin] (fp32) += gradient of tsp_conv_fprop's weights given its input x and dy.  The caller zeroes dw
// (or keeps a running sum in it: micro-batches accumulate).
int tsp_conv_wgrad(const void* x, const void* dy, float* dw, int n, int h, int w, int cin, int cout, int k, int s,
                   int* status, cudaStream_t stream) {
  if (!shape_ok(n, h, w, cin, cout, k, s)) return -3;
  if (((uintptr_t)x | (uintptr_t)dy) & 15) return -2;
  // A 1x1 stride-1 convolution is a linear layer over its pixels.  The CTA-pair product's tile is 256 output channels high:
  // where it is full it is faster at every size tried (B200, 256 images: 64 -> 256 at 56 x 56 79 us against 84, 512 -> 256
  // at 28 x 28 54 / 67, 1024 -> 256 at 14 x 14 29 / 39, 512 -> 2048 at 7 x 7 28 / 39; 37 images: 11 - 16 / 20 - 23); with
  // 64 or 128 output channels it is not (256 -> 64 at 56 x 56 86 / 79).
  if (k == 1 && s == 1 && cout % 256 == 0 && ((uintptr_t)dw & 15) == 0) {
    const void* const dys[1] = {dy};
    return tsp_gemm_bf16_wgrad_2cta(dys, 1, x, dw, cout, cin, n * h * w, cout, cin, cin, status, stream);
  }
  if (cin == 64 && cout == 64 && halo_applies(k, s, w, h)) return launch_wgrad_halo(x, dy, dw, n, h, w, status, stream);
  const int bn = cout % 256 == 0 ? 256 : (cout % 128 == 0 ? 128 : 64);
  Plan p = plan_input(x, n, h, w, cin, k, s, bn == 256 ? 64 : 128);
  if (!p.ok) return -6;
  Geom& g = p.g;
  const int pad = (k - 1) / 2, ho = (h + 2 * pad - k) / s + 1, wo = (w + 2 * pad - k) / s + 1;
  g.nc = cout;
  g.ldw = k * k * cin;
  const bool flat = k == 1 && s == 1;
  CUtensorMap dymap;
  const bool ok = flat ? act_map(&dymap, dy, cout, g.out_w, 1, 1, cout, (int64_t)cout * g.out_w, (int64_t)cout * g.out_w,
                                 g.box_w, 1, 1)
                       : act_map(&dymap, dy, cout, wo, ho, n, cout, (int64_t)wo * cout, (int64_t)ho * wo * cout, g.box_w,
                                 g.box_h, g.box_n);
  if (!ok) return -6;
  // Work items = output tiles x pieces of the pixel range; about two items per SM and never a handful more than a
  // multiple of the SM count (those would cost a whole extra round).
  const int m_tiles = (g.n_taps * (cin / 64) + 1) / 2, n_tiles = (cout + bn - 1) / bn;
  const int tiles = m_tiles * n_tiles, boxes = g.tiles_w * g.tiles_h * g.tiles_n;
  int splits = 2 * sm_count() / tiles;
  if (splits > boxes) splits = boxes;
  if (splits < 1) splits = 1;
  g.splits = splits;
  if (bn == 256) return launch_wgrad<256>(p, dymap, dw, status, stream);
  if (bn == 128) return launch_wgrad<128>(p, dymap, dw, status, stream);
  return launch_wgrad<64>(p, dymap, dw, status, stream);
}

}  // extern "C"

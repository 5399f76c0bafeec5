// bf16 GEMM with two SMs per output tile: C[M,N] = A[M,K] * B[N,K]^T, fp32 accumulation, 256 x BN tiles (BN = 256, 128
// or 64, see pick_bn).
//
// A cluster of two CTAs owns one 256 x BN tile (figures for BN = 256).  CTA r of the pair loads rows [128 r, 128 r + 128) of the A tile and
// rows [128 r, 128 r + 128) of the B tile (half of N) with its own TMA loads; the leader CTA (rank 0) issues
// tcgen05.mma.cta_group::2, which reads A from both CTAs' shared memory and the two halves of B, and writes each
// CTA's 128 x 256 accumulator slice into that CTA's tensor memory.  Compared with the one-CTA kernel
// (gemm_tcgen05.cu: 48 KB of operands per 128 x 256 x 64 step) each SM moves 32 KB per step for the same FLOPs.
//
// Synchronisation (all mbarriers; every wait bounded in time, see tc5::mbar_wait):
//   full[s]        in the leader: armed by the leader's producer with the bytes of BOTH CTAs; every TMA load of the
//                  pair completes its bytes on the leader's barrier (cp.async.bulk.tensor ... .cta_group::2);
//   empty[g]       in each CTA, one per GROUP of two slots: after the MMAs of a group's second slot the leader issues
//                  ONE tcgen05.commit that arrives on the barrier of both CTAs (a commit costs the issuing thread as
//                  much as several MMA issues; two per k-block made the issuing thread, not the tensor core, the limit);
//   tmem_full[a]   in each CTA: committed by the leader (to both CTAs at once) after the last MMA of a tile;
//   tmem_empty[a]  in the leader: one arrival per epilogue warp of the pair (the peer's arrive remotely).
// Epilogue: TMEM -> registers -> swizzled shared memory -> TMA store (32 rows x 128 bytes per store, two buffers
// per warp); direct per-thread stores when C has no 16-byte-aligned base and row pitch.
// The cluster is synchronised once after barrier initialisation and once before exit, so no CTA leaves while its
// partner can still touch its shared memory.
#include <cuda.h>

#include "gelu.cuh"
#include "tcgen05.cuh"
#include "tspipe_kernels.h"

extern int g_tsp_sm_reserve;          // defined in peer.cu

namespace {

constexpr int BM = 128;          // rows per CTA (pair tile: 256)
constexpr int BK = 64;
constexpr int UMMA_K = 16;
constexpr uint64_t kWaitNs = 2000000000ull;   // every mbarrier wait gives up after two seconds
constexpr int kGroup = 2;                       // stages released per tcgen05.commit
constexpr int kABytes = BM * BK * 2;
constexpr int kStoreBytes = 8 * 32 * 128;                       // two 32 x 128 byte blocks per epilogue warp, or 16 of 32 x 64
// BN = tile columns (256, 128 or 64); each CTA stages BN / 2 rows of B
template <int BN> struct Cfg {
  static constexpr int kStages = BN == 256 ? 6 : 8;
  static constexpr int kGroups = kStages / kGroup;
  static constexpr int kBBytes = (BN / 2) * BK * 2;
  static constexpr int kStageBytes = kABytes + kBBytes;         // per CTA
  static constexpr int kTmemCols = 2 * BN;                      // two accumulator buffers
  static constexpr int kSmemBytes = kStages * kStageBytes + kStoreBytes + 1024 + 256;
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// shared::cluster address of the same shared-memory offset in CTA `rank` of this cluster
__device__ __forceinline__ uint32_t map_to_cta(uint32_t local_addr, uint32_t rank) {
  uint32_t out;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(out) : "r"(local_addr), "r"(rank));
  return out;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// TMA load into this CTA's shared memory whose byte count completes on a barrier of the pair's leader.
__device__ __forceinline__ void tma_load_2d_pair(void* smem_dst, const CUtensorMap* map, uint32_t leader_bar, int x,
                                                 int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], "
      "[%2];" ::"r"(smem_u32(smem_dst)),
      "l"(map), "r"(leader_bar), "r"(x), "r"(y)
      : "memory");
}

// one commit that arrives on the barrier at the same shared-memory offset in BOTH CTAs of the pair (a commit costs
// the issuing thread as much as several MMA issues, so the pair is signalled with one instruction, not two)
__device__ __forceinline__ void umma_commit_pair_both(uint32_t local_bar_addr) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
               ::"r"(local_bar_addr), "h"((uint16_t)3)
               : "memory");
}
__device__ __forceinline__ void umma_bf16_pair_lo(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t idesc,
                                                  uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\t"
      "setp.ne.b32 p, %5, 0;\n\t"
      "mov.b64 da, {%1, %3};\n\t"
      "mov.b64 db, {%2, %3};\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], da, db, %4, p;\n\t}"
      ::"r"(d_tmem), "r"(a_lo), "r"(b_lo), "r"(tc5::kDescHi), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void tmem_ld_32x32_issue(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// TMA store of one 32-row x 128-byte block (128-byte swizzle) from shared memory; rows / columns beyond the
// tensor's extent are clipped by the hardware.
__device__ __forceinline__ void tma_store_2d(const CUtensorMap* map, const void* smem_src, int x, int y) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];" ::"l"(map),
               "r"(smem_u32(smem_src)), "r"(x), "r"(y)
               : "memory");
  asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}
// The same block added element by element to what is in memory (fp32), in L2.
__device__ __forceinline__ void tma_reduce_add_2d(const CUtensorMap* map, const void* smem_src, int x, int y) {
  asm volatile("cp.reduce.async.bulk.tensor.2d.global.shared::cta.add.tile.bulk_group [%0, {%2, %3}], [%1];" ::"l"(map),
               "r"(smem_u32(smem_src)), "r"(x), "r"(y)
               : "memory");
  asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}
__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
  __nv_bfloat162 t = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&t);
}

__device__ __forceinline__ float gelu_erf(float x) { return 0.5f * x * (1.f + erff(x * 0.70710678118654752f)); }

// The three products of a linear layer.  An operand whose contraction index is the slow one in memory is staged as boxes
// of 64 contraction rows x 64 columns and read by the tensor core as an MN-major tile: no transposed copy exists anywhere.
enum Kind {
  kTN = 0,      // C = A[m, k] B[n, k]^T      forward
  kNN = 1,      // C = A[m, k] B[k, n]        gradient of the input; A may be up to three matrices side by side along k
  kGelu = 3,    // C0 = A[m, k] B[n, k]^T rounded, C1 = gelu(C0 + bias): the first half of an MLP; C0 only where a backward needs it
  kRed = 2      // C += A[k, m]^T B[k, n]     gradient of the weight: fp32, split along k, added in L2 by the TMA unit; A may
                //                            be up to three matrices side by side along m
};
// Epilogue warps: four per TMEM lane quarter where the epilogue computes.  The GELUs of a tile are about as many issue slots as
// the products of a K = 768 tile are clocks, so that the warps of a scheduler have to cover each other's waits for TMEM, the
// reciprocal and the exponential; with two per quarter they did not.  Each stages 32 x 32 blocks in a buffer of its own, which
// keeps the staging at 32 KB.  B200, 12608 x 3072 x 768, both outputs: 74.8 us with two -> 70.7, 16384 rows and one output
// 83.0 -> 78.8.  With few tiles the larger start costs nothing that shows: 128 rows 15.4 and 15.4, 788 21.5 and 20.5, 1576 25.5 and 23.6; 4096
// x 1024 of 128 rows 16.5 both, of 788 23.5 and 22.6; 1536 x 384 13.3 and 13.3, 15.3 and 15.3.
__host__ __device__ constexpr int epi_warps(int kind) { return kind == kGelu ? 16 : 4; }
// bytes of a row of C that a warp stages and stores at a time
__host__ __device__ constexpr int block_bytes(int kind) { return kind == kGelu ? 64 : 128; }
constexpr int kMaxASrc = 3;
struct AMaps {
  CUtensorMap m[kMaxASrc];
};
// Where the columns of C go: with kTN up to three matrices of n_per columns side by side (a fused projection whose
// blocks are wanted apart), n_per a multiple of 64.
constexpr int kMaxCDst = 3;
struct CMaps {
  CUtensorMap m[kMaxCDst];
};

template <typename OutT, bool STATS, int BN, int KIND>
__global__ void __launch_bounds__(64 + 32 * epi_warps(KIND), 1)
gemm_tcgen05_2cta_kernel(const __grid_constant__ AMaps tmap_a, int a_per, const __grid_constant__ CUtensorMap tmap_b,
                         const __grid_constant__ CMaps tmap_c, int n_per, int tma_store, OutT* __restrict__ c,
                         const float* __restrict__ bias, int m, int n, int k, int ldc, int epi, int splits,
                         float* __restrict__ col_sums, int seg_rows, int* __restrict__ status) {
  using C = Cfg<BN>;
  constexpr int kStages = C::kStages, kGroups = C::kGroups, kStageBytes = C::kStageBytes, kTmemCols = C::kTmemCols;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* tiles = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint8_t* store_bufs = tiles + kStages * kStageBytes; // 1024-aligned: the swizzle pattern follows address bits
  uint64_t* bars = (uint64_t*)(store_bufs + kStoreBytes);
  uint64_t* full_bar = bars;                           // [kStages]  used in the leader only
  uint64_t* empty_bar = bars + kStages;                // [kStages]  in each CTA
  uint64_t* tmem_full_bar = bars + 2 * kStages;        // [2]        in each CTA
  uint64_t* tmem_empty_bar = bars + 2 * kStages + 2;   // [2]        used in the leader only
  uint32_t* tmem_slot = (uint32_t*)(bars + 2 * kStages + 4);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const bool leader = rank == 0;
  const int pair = blockIdx.x >> 1, num_pairs = gridDim.x >> 1;
  const int tiles_m = (m + 2 * BM - 1) / (2 * BM), tiles_n = (n + BN - 1) / BN;
  const int num_tiles = tiles_m * tiles_n;
  const int num_kb = (k + BK - 1) / BK;
  // work items: tiles, and with kRed each tile in `splits` pieces of the contraction (item = piece * num_tiles + tile)
  // otherwise the tiles of the last, partial round in `splits` pieces of their columns each, side by side on the idle pairs
  const int whole = KIND == kRed ? 0 : num_tiles / num_pairs * num_pairs;
  const int num_items = whole + (num_tiles - whole) * splits;
  int width = BN;                                      // columns of the item at hand, and its first one within the tile
  int first_col = 0;
  auto item_range = [&](int t, int& tile, int& kb_lo, int& kb_hi) {
    if constexpr (KIND == kRed) {
      const int sp = t / num_tiles;
      tile = t - sp * num_tiles;
      kb_lo = (int)((int64_t)num_kb * sp / splits);
      kb_hi = (int)((int64_t)num_kb * (sp + 1) / splits);
    } else {
      tile = t; kb_lo = 0; kb_hi = num_kb;
      if (t >= whole) {
        const int j = t - whole;
        tile = whole + j / splits;
        width = BN / splits;
        first_col = j % splits * width;
      }
    }
  };

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(full_bar + s, 1);
      mbar_init(empty_bar + s, 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(tmem_full_bar + a, 1);
      mbar_init(tmem_empty_bar + a, 2 * epi_warps(KIND));
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&tmap_a.m[0]) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&tmap_b) : "memory");
  }
  if (warp == 1) {        // warp 1 of BOTH CTAs: paired allocation of both accumulator buffers
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"((uint32_t)kTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  cluster_sync_all();                                   // both CTAs' barriers exist before anyone signals them
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = *tmem_slot;
  tsp::wait_for_previous();
  bias = tsp::written(bias);

  if (warp == 0) {
    // ---------------- TMA producer (one thread per CTA) ----------------
    if (lane == 0) {
      uint32_t it = 0;
      bool ok = true;
      for (int t = pair; t < num_items && ok; t += num_pairs) {
        // N tiles fastest: the pairs that run together share rows of A (read from DRAM once, then from L2) and sweep
        // the weights, which stay in L2; walking all of M per N tile would stream A from DRAM once per N tile
        int tile, kb_lo, kb_hi;
        item_range(t, tile, kb_lo, kb_hi);
        const int m0 = (tile / tiles_n) * 2 * BM + (int)rank * BM;
        const int n0 = (tile % tiles_n) * BN + first_col + (int)rank * (width / 2);    // (a narrow item's box holds more than it uses)
        for (int kb = kb_lo; kb < kb_hi; ++kb, ++it) {
          const int s = it % kStages;
          if (it % kGroup == 0) {                 // first stage of a group: the whole group must have been released
            const uint32_t grp = (it / kGroup) % kGroups, round = (it / kGroup) / kGroups;
            if (round > 0 && !tc5::mbar_wait_parked(empty_bar + grp, (round - 1) & 1, status, 1, kWaitNs)) { ok = false; break; }
          }
          uint8_t* a_dst = tiles + s * kStageBytes;
          uint8_t* b_dst = a_dst + kABytes;
          if (leader) mbar_expect_tx(full_bar + s, 2u * (uint32_t)kStageBytes);
          const uint32_t lbar = map_to_cta(smem_u32(full_bar + s), 0);
          if constexpr (KIND == kRed) {
#pragma unroll
            for (int j = 0; j < BM / 64; ++j) {        // a_per: columns per source; past the last one reads as zeros
              const int col = m0 + j * 64, src = min(col / a_per, (m - 1) / a_per);
              tma_load_2d_pair(a_dst + j * 8192, &tmap_a.m[src], lbar, col - src * a_per, kb * BK);
            }
          } else if constexpr (KIND == kNN) {
            const int src = kb / a_per;                // k blocks per source
            tma_load_2d_pair(a_dst, &tmap_a.m[src], lbar, (kb - src * a_per) * BK, m0);
          } else {
            tma_load_2d_pair(a_dst, &tmap_a.m[0], lbar, kb * BK, m0);
          }
          if constexpr (KIND == kTN || KIND == kGelu) {
            tma_load_2d_pair(b_dst, &tmap_b, lbar, kb * BK, n0);
          } else {
#pragma unroll
            for (int j = 0; j < BN / 128; ++j) tma_load_2d_pair(b_dst + j * 8192, &tmap_b, lbar, n0 + j * 64, kb * BK);
          }
        }
      }
      tsp::let_next_start();
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer (leader CTA only) ----------------
    if (leader) {
      const bool issuer = tc5::elect_one();
      auto arrived = [&](uint64_t* bar, uint32_t parity, int code) -> bool {      // the same for the warp
        return __all_sync(0xffffffffu, tc5::mbar_wait(bar, parity, status, code, kWaitNs)) != 0;
      };
      constexpr bool kAmn = KIND == kRed, kBmn = KIND == kNN || KIND == kRed;
      static_assert(!kBmn || BN % 128 == 0, "an MN-major half tile of B is whole 64-column boxes");
      const uint32_t tiles_addr = smem_u32(tiles);
      uint32_t it = 0, lt = 0;
      bool ok = true;
      for (int t = pair; t < num_items && ok; t += num_pairs, ++lt) {
        int tile, kb_lo, kb_hi;
        item_range(t, tile, kb_lo, kb_hi);
        const uint32_t acc = lt & 1, use = lt >> 1;
        if (use > 0) {
          ok = arrived(tmem_empty_bar + acc, (use - 1) & 1, 4);
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        }
        const uint32_t d_tmem = tmem_base + acc * BN, idesc = tc5::make_idesc(2 * BM, width, kAmn, kBmn);
        uint32_t accum = 0u;
        for (int kb = kb_lo; kb < kb_hi; ++kb, ++it) {
          const int s = it % kStages;
          const uint32_t round = it / kStages;
          ok = arrived(full_bar + s, round & 1, 2);
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t a_addr = tiles_addr + s * kStageBytes;
          const uint32_t a_lo = kAmn ? tc5::desc_lo_mn_major(a_addr, 8192) : tc5::desc_lo_k_major(a_addr);
          const uint32_t b_lo = kBmn ? tc5::desc_lo_mn_major(a_addr + kABytes, 8192) : tc5::desc_lo_k_major(a_addr + kABytes);
#pragma unroll
          for (int kk = 0; kk < BK / UMMA_K; ++kk) {  // 16 along K: +32 bytes in a K-major row, +2048 bytes (16 rows) MN-major
            if (issuer) umma_bf16_pair_lo(d_tmem, a_lo + (kAmn ? 128 : 2) * kk, b_lo + (kBmn ? 128 : 2) * kk, idesc, accum);
            accum = 1u;
          }
          // the group's slots are free again in both CTAs once these MMAs have read them
          if (issuer && it % kGroup == kGroup - 1) umma_commit_pair_both(smem_u32(empty_bar + (it / kGroup) % kGroups));
        }
        if (issuer) umma_commit_pair_both(smem_u32(tmem_full_bar + acc));
      }
    }
  } else {
    // ---------------- epilogue (both CTAs): this CTA's 128 rows, all BN columns ----------------
    // Per warp: 32 accumulator rows.  Blocks of 128 output bytes per row (64 bf16 or 32 fp32 columns; kGelu 64 bytes) go
    // TMEM -> registers -> (bias, GELU, convert) -> swizzled shared memory -> one TMA store; two staging
    // buffers per warp, so the store of block i overlaps the conversion of block i + 1 (kGelu one).  Without a usable
    // tensor map for C (unaligned base or row pitch) every thread stores its own row directly.
    constexpr int kRowBytes = block_bytes(KIND), kStoreBufBytes = 32 * kRowBytes, kCols = kRowBytes / (int)sizeof(OutT);
    constexpr int kBufs = kStoreBytes / kStoreBufBytes / epi_warps(KIND);         // staging buffers per warp
    const int quarter = warp & 3, group = (warp - 2) >> 2;
    uint8_t* my_bufs = store_bufs + (warp - 2) * kBufs * kStoreBufBytes;
    uint32_t lt = 0, nstore = 0;
    bool ok = true;
    // STATS: per-column sum and sum of squares of the rounded outputs (the statistics of a BatchNorm that
    // follows a 1x1 convolution), kept in registers while this warp stays in the same column block and row
    // group: cs[i] = {sum, sumsq of column 2*lane, sum, sumsq of column 2*lane+1} of 64-column block i.
    float cs[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) { cs[i][0] = cs[i][1] = cs[i][2] = cs[i][3] = 0.f; }
    int cur_n0 = -1, cur_seg = 0;
    auto flush_stats = [&]() {
      if (cur_n0 >= 0) {
        float* dst = col_sums + (int64_t)cur_seg * 2 * n;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int col = cur_n0 + 64 * i + 2 * lane;
          if (col < n) { atomicAdd(dst + col, cs[i][0]); atomicAdd(dst + n + col, cs[i][1]); }
          if (col + 1 < n) { atomicAdd(dst + col + 1, cs[i][2]); atomicAdd(dst + n + col + 1, cs[i][3]); }
          cs[i][0] = cs[i][1] = cs[i][2] = cs[i][3] = 0.f;
        }
      }
    };
    for (int t = pair; t < num_items && ok; t += num_pairs, ++lt) {
      int tile, kb_lo, kb_hi;
      item_range(t, tile, kb_lo, kb_hi);
      const int m0 = (tile / tiles_n) * 2 * BM + (int)rank * BM, n0 = (tile % tiles_n) * BN + first_col;
      const uint32_t acc = lt & 1, use = lt >> 1;
      if (STATS) {
        const int seg = m0 / seg_rows;
        if (n0 != cur_n0 || seg != cur_seg) { flush_stats(); cur_n0 = n0; cur_seg = seg; }
      }
      ok = tc5::mbar_wait_warp(tmem_full_bar + acc, use & 1, status, 3, kWaitNs, lane);   // one way out per warp
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      bool live = true;                            // after a wait that ran out the accumulator may hold part of its sum
      if constexpr (KIND == kRed) live = *((volatile int*)status) == 0;
      const int row0 = m0 + quarter * 32, row = row0 + lane;
      // the block's values -> swizzled staging buffer -> TMA store at column x of `map`; returns the buffer
      auto stage = [&](const float (&v)[kCols], const CUtensorMap* map, int x, bool inside) -> uint8_t* {
        uint8_t* buf = my_bufs + (nstore % kBufs) * kStoreBufBytes;
        if (nstore >= kBufs) {       // the store issued kBufs blocks ago has finished reading this buffer
          if (lane == 0) {
            if constexpr (kBufs == 2) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
            else asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
          }
          __syncwarp();
        }
        uint8_t* my_row = buf + lane * kRowBytes;
        const int swizzle = kRowBytes == 128 ? lane & 7 : (lane >> 1) & 3;
#pragma unroll
        for (int j = 0; j < kRowBytes / 16; ++j) {   // 16-byte piece j of this row sits at piece (j ^ swizzle)
          uint4 q;
          if constexpr (sizeof(OutT) == 2) {
            q.x = pack_bf16x2(v[8 * j + 0], v[8 * j + 1]);
            q.y = pack_bf16x2(v[8 * j + 2], v[8 * j + 3]);
            q.z = pack_bf16x2(v[8 * j + 4], v[8 * j + 5]);
            q.w = pack_bf16x2(v[8 * j + 6], v[8 * j + 7]);
          } else {
            q.x = __float_as_uint(v[4 * j + 0]);
            q.y = __float_as_uint(v[4 * j + 1]);
            q.z = __float_as_uint(v[4 * j + 2]);
            q.w = __float_as_uint(v[4 * j + 3]);
          }
          *reinterpret_cast<uint4*>(my_row + ((j ^ swizzle) << 4)) = q;
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0) {
          if (!inside) asm volatile("cp.async.bulk.commit_group;" ::: "memory");     // keep the group count in step
          else if constexpr (KIND == kRed) tma_reduce_add_2d(map, buf, x, row0);
          else tma_store_2d(map, buf, x, row0);
        }
        ++nstore;
        return buf;
      };
      // one block of kCols columns; returns false past the matrix edge
      auto chunk = [&](int c0, float* st) -> bool {
        if (n0 + c0 >= n) return false;            // columns past the matrix edge: nothing to convert or store
        float v[kCols];
        {
          uint32_t r[kCols];
          const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + acc * BN + (uint32_t)c0;
          tmem_ld_32x32_issue(taddr, r);
          if constexpr (kCols == 64) tmem_ld_32x32_issue(taddr + 32, r + 32);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < kCols; ++j) v[j] = __uint_as_float(r[j]);
        }
        const int col = n0 + c0;
        if constexpr (KIND == kGelu) {             // n is a multiple of 64, C is written by the TMA unit
          const bool inside = row0 < m;
          tsp::round_as<OutT>(v);
          if (epi != 0) stage(v, &tmap_c.m[0], col, inside);
          const float4* bp = reinterpret_cast<const float4*>(bias + col);
#pragma unroll
          for (int j = 0; j < kCols / 4; ++j) {
            const float4 b4 = __ldg(bp + j);
            static_assert(sizeof(OutT) == 2, "two values an instruction");
            tsp::gelu2(tsp::Pair(v[4 * j + 0], v[4 * j + 1]) + tsp::Pair(b4.x, b4.y)).split(v[4 * j + 0], v[4 * j + 1]);
            tsp::gelu2(tsp::Pair(v[4 * j + 2], v[4 * j + 3]) + tsp::Pair(b4.z, b4.w)).split(v[4 * j + 2], v[4 * j + 3]);
          }
          stage(v, &tmap_c.m[1], col, inside);
          return true;
        }
        if (epi != 0 && col < n) {
          if (col + kCols <= n && (((uintptr_t)(bias + col)) & 15) == 0) {
            // whole block inside the matrix: the block's bias values as 16-byte loads (every lane reads the same
            // addresses, one broadcast transaction each) instead of one scalar load per element
            const float4* bp = reinterpret_cast<const float4*>(bias + col);
#pragma unroll
            for (int j = 0; j < kCols / 4; ++j) {
              const float4 b4 = __ldg(bp + j);
              v[4 * j + 0] += b4.x; v[4 * j + 1] += b4.y; v[4 * j + 2] += b4.z; v[4 * j + 3] += b4.w;
            }
          } else {
#pragma unroll
            for (int j = 0; j < kCols; ++j) v[j] += (col + j < n) ? bias[col + j] : 0.f;
          }
          if (epi == 2) {
#pragma unroll
            for (int j = 0; j < kCols; ++j) v[j] = gelu_erf(v[j]);
          }
        }
        if (tma_store) {
          const int dst = KIND == kTN ? col / n_per : 0;
          const uint8_t* buf = stage(v, &tmap_c.m[dst], col - dst * n_per, live && row0 < m && col < n);
          if (STATS && st != nullptr) {
            // column sums of the staged (rounded) block: lane owns columns 2*lane, 2*lane+1; rows past the
            // matrix edge hold exact zeros (their A rows were zero-filled)
#pragma unroll 8
            for (int rr = 0; rr < 32; ++rr) {
              const uint32_t wv = *reinterpret_cast<const uint32_t*>(buf + rr * 128 + (((lane >> 2) ^ (rr & 7)) << 4) +
                                                                     (lane & 3) * 4);
              const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&wv));
              st[0] += f.x; st[1] += f.x * f.x; st[2] += f.y; st[3] += f.y * f.y;
            }
          }
        } else if (row < m && col < n) {
          OutT* dst = c + (int64_t)row * ldc + col;
#pragma unroll
          for (int j = 0; j < kCols; ++j)       // constant indices only: v stays in registers
            if (col + j < n) tsp::st(dst, j, v[j]);
        }
        return true;
      };
      if constexpr (STATS) {
        static_assert(!STATS || (kCols == 64 && BN == 256), "column statistics are kept for bf16 outputs and the widest tile");
        if (chunk(0, cs[0]) && chunk(64, cs[1]) && chunk(128, cs[2])) chunk(192, cs[3]);
      } else {
#pragma unroll 1
        for (int c0 = KIND == kGelu ? group * kCols : 0; c0 < width; c0 += kCols * (epi_warps(KIND) / 4))
          if (!chunk(c0, nullptr)) break;
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(map_to_cta(smem_u32(tmem_empty_bar + acc), 0));
    }
    if (STATS) flush_stats();
    if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");   // staging buffers are free again
    __syncwarp();
  }
  if (*((volatile int*)status) != 0) {
    // a wait ran out somewhere: give TMA loads and MMAs that are still in flight time to land before the pair's
    // shared memory and tensor memory are released
    for (int i = 0; i < 64; ++i) __nanosleep(1000);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  cluster_sync_all();                                   // nobody touches the partner's memory after this point
  if (warp == 1) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)kTmemCols)
                 : "memory");
  }
}

bool make_map(CUtensorMap* map, const void* ptr, int rows, int cols, int ld, int box_rows) {
  const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows}, strides[1] = {(cuuint64_t)ld * 2};
  const cuuint32_t box[2] = {(cuuint32_t)BK, (cuuint32_t)box_rows};
  return tc5::encode_tiled(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, ptr, 2, dims, strides, box,
                           CU_TENSOR_MAP_L2_PROMOTION_L2_256B);
}

bool make_store_map(CUtensorMap* map, void* ptr, int rows, int cols, int ld, bool bf16, int row_bytes) {
  const int esz = bf16 ? 2 : 4;
  const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows}, strides[1] = {(cuuint64_t)ld * esz};
  const cuuint32_t box[2] = {(cuuint32_t)(row_bytes / esz), 32};
  return tc5::encode_tiled(map, bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, ptr, 2, dims,
                           strides, box, CU_TENSOR_MAP_L2_PROMOTION_NONE,
                           row_bytes == 128 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B);
}

// About the clocks that a pair needs for 64 rows of a weight gradient's contraction, and what an item costs besides: its
// accumulator goes out as fp32 additions.  B200, 768 x 768 x 12608: 82 us in one piece per tile (197 steps), 18.6 in 8, 20.4 in 16;
// over 22 shapes of linear layers and 1x1 convolutions the choice is the fastest of those tried or within 5 percent of it,
// and is the same with 640 clocks.
constexpr int kBlockClocks = 740, kRedClocks = 3000;

// Tile width: 256 columns, halved while all tiles of the narrower width still run at once.  A step is bound by the
// operands' way from L2, so a narrower tile does not pay for a fuller last wave (12608 x 3072 x 768, B200: 46.7 us at 256
// columns, 54.9 at 128, 89.0 at 64), but shorter tiles on more SMs do where the wide ones leave the chip idle
// (788 x 768 x 768: 9.9 us at 256, 8.7 at 64; 256 x 4096 x 2048 15.5 and 11.8, 256 x 256 x 4096 23.3 and 16.8).
int pick_bn(int m, int n, int pairs, int least) {
  const int64_t tiles_m = (m + 2 * BM - 1) / (2 * BM);
  int bn = 256;
  while (bn > least && tiles_m * ((n + bn / 2 - 1) / (bn / 2)) <= pairs) bn /= 2;
  return bn;
}

// Pieces of the contraction of a weight gradient: the number that finishes soonest by these clocks.
int pick_splits(int m, int n, int k, int bn, int pairs) {
  const int64_t tiles = (int64_t)((m + 2 * BM - 1) / (2 * BM)) * ((n + bn - 1) / bn), kb = (k + BK - 1) / BK;
  int best = 1;
  int64_t best_cost = 0;
  for (int sp = 1; sp <= kb && (sp == 1 || tiles * sp <= 2 * pairs); ++sp) {
    const int64_t cost = (tiles * sp + pairs - 1) / pairs * ((kb + sp - 1) / sp * kBlockClocks + kRedClocks);
    if (sp == 1 || cost < best_cost) { best = sp; best_cost = cost; }
  }
  return best;
}

// Pieces of a tile's columns in the last round of tiles, where it leaves at least half of the pairs idle: as many as `most` and
// as run at once.  A step of a narrow piece takes less time, and the sums are formed in the same order.  12608 x 768 (150 tiles on 74
// pairs), B200: K = 3072 56.5 us with whole tiles in the third round, 47.8 in quarters; in halves (MN-major B) 53.8.  Within a
// ViT-B block 880 us and 877.
int last_round_pieces(int tiles, int pairs, int most) {
  const int left = tiles % pairs;
  int pieces = 1;
  if (tiles > pairs && left != 0)
    while (2 * pieces <= most && 2 * pieces * left <= pairs) pieces *= 2;
  return pieces;
}

struct Args {
  const void* a[kMaxASrc];
  int n_src;                    // matrices side by side, each k / n_src (kNN) or m / n_src (kRed) wide
  const void* b;
  void* c[kMaxCDst];
  int n_dst;                    // matrices side by side along n, each n / n_dst wide (kTN, through the TMA unit only)
  const float* bias;
  int m, n, k, lda, ldb, ldc, epi;
  float* col_sums;
  int seg_rows;
  int* status;
};

template <typename OutT, bool STATS, int BN, int KIND>
int launch_bn(const Args& p, int dev, int max_pairs, cudaStream_t stream) {
  constexpr int kSmemBytes = Cfg<BN>::kSmemBytes;
  AMaps ta;
  CUtensorMap tb;
  const int a_src = (KIND == kRed ? p.m : p.k) / p.n_src;
  for (int i = 0; i < kMaxASrc; ++i) {
    if (i >= p.n_src) { ta.m[i] = ta.m[0]; continue; }
    const void* a = p.a[i];
    if (!(KIND == kRed ? make_map(&ta.m[i], a, p.k, a_src, p.lda, 64) : make_map(&ta.m[i], a, p.m, a_src, p.lda, BM))) return -6;
  }
  constexpr bool kBmn = KIND == kNN || KIND == kRed;
  if (!(kBmn ? make_map(&tb, p.b, p.k, p.n, p.ldb, 64) : make_map(&tb, p.b, p.n, p.k, p.ldb, BN / 2))) return -6;
  CMaps tc;
  const int n_per = KIND == kGelu ? p.n : p.n / p.n_dst;
  int tma_store = 1;
  for (int i = 0; i < kMaxCDst; ++i) {
    if (i >= p.n_dst) { tc.m[i] = tc.m[0]; continue; }
    void* c = p.c[i];
    if (c == nullptr) c = p.c[1];                       // (kGelu without C0)
    tc.m[i] = tb;               // placeholder when C cannot be described (the kernel then stores directly)
    if ((((uintptr_t)c & 15) != 0) || ((p.ldc * (int)sizeof(OutT)) % 16 != 0) ||
        !make_store_map(&tc.m[i], c, p.m, n_per, p.ldc, sizeof(OutT) == 2, block_bytes(KIND)))
      tma_store = 0;
  }
  // statistics come from the staged blocks, sums and several destinations need the TMA unit
  if ((STATS || KIND == kRed || p.n_dst > 1) && !tma_store) return -3;
  auto kern = gemm_tcgen05_2cta_kernel<OutT, STATS, BN, KIND>;
  static bool attr_set[64] = {};
  if (!attr_set[dev]) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes);
    if (e != cudaSuccess) return (int)e;
    attr_set[dev] = true;
  }
  const int num_tiles = ((p.n + BN - 1) / BN) * ((p.m + 2 * BM - 1) / (2 * BM));
  const int splits = KIND == kRed ? pick_splits(p.m, p.n, p.k, BN, max_pairs)
                                  : (STATS ? 1 : last_round_pieces(num_tiles, max_pairs, BN / (kBmn ? 128 : 64)));
  const int num_items = KIND == kRed ? num_tiles * splits : num_tiles;
  const int pairs = max_pairs > num_items ? num_items : max_pairs;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2 * pairs, 1, 1);
  cfg.blockDim = dim3(64 + 32 * epi_warps(KIND), 1, 1);
  cfg.dynamicSmemBytes = kSmemBytes;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1] = tsp::early_start();
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  cudaError_t e = cudaLaunchKernelEx(&cfg, kern, ta, p.n_src > 1 ? (KIND == kRed ? a_src : a_src / BK) : 0x7fffffff, tb, tc, KIND == kTN && p.n_dst > 1 ? n_per : 0x7fffffff, tma_store,
                                     (OutT*)p.c[0], p.bias,
                                     p.m, p.n, p.k, p.ldc, p.epi, splits, p.col_sums, p.seg_rows, p.status);
  return (int)e;
}

template <typename OutT, bool STATS, int KIND = kTN>
int launch(const Args& p, cudaStream_t stream) {
  static int n_sm[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  dev &= 63;
  if (n_sm[dev] == 0) {
    int v = 0;
    cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev);
    n_sm[dev] = v > 0 ? v : 148;
  }
  int pairs = (n_sm[dev] - g_tsp_sm_reserve) / 2;      // SMs left to communication kernels stay free
  if (pairs < 4) pairs = 4;
  if constexpr (KIND == kRed) {
    // the contraction is split until the chip is full, so the width only matters where the output is narrower
    return p.n > 128 ? launch_bn<OutT, STATS, 256, KIND>(p, dev, pairs, stream)
                     : launch_bn<OutT, STATS, 128, KIND>(p, dev, pairs, stream);
  } else if constexpr (!STATS) {
    const int bn = pick_bn(p.m, p.n, pairs, KIND == kNN ? 128 : 64);   // MN-major B: halves of whole 64-column boxes
    if constexpr (KIND != kNN) {
      if (bn == 64) return launch_bn<OutT, STATS, 64, KIND>(p, dev, pairs, stream);
    }
    if (bn == 128) return launch_bn<OutT, STATS, 128, KIND>(p, dev, pairs, stream);
    return launch_bn<OutT, STATS, 256, KIND>(p, dev, pairs, stream);
  } else {
    return launch_bn<OutT, STATS, 256, KIND>(p, dev, pairs, stream);
  }
}

}  // namespace

extern "C" {

// Two-SM variant of tsp_gemm_bf16_tn, same arguments: C[m,n] = A[m,k] * B[n,k]^T (+ bias[n]) (-> GELU), bf16
// operands, C bf16 or fp32; epi 0 none, 1 bias, 2 bias + GELU.
// `status`: one zeroed int in device memory; non-zero afterwards = a bounded wait ran out (1 producer, 2 MMA on
// operands, 3 epilogue, 4 MMA on a free accumulator) and C is not valid.
int tsp_gemm_bf16_tn_2cta(const void* a, const void* b, void* c, const float* bias, int m, int n, int k, int lda,
                          int ldb, int ldc, int out_dtype, int epi, int* status, cudaStream_t stream) {
  if (m <= 0 || n <= 0 || k <= 0) return 0;
  if (epi != 0 && bias == nullptr) return -3;
  if ((lda % 8) || (ldb % 8) || (k % 8)) return -3;
  if (((uintptr_t)a | (uintptr_t)b) & 15) return -2;
  const Args p = {{a, nullptr, nullptr}, 1, b, {c, nullptr, nullptr}, 1, bias, m, n, k, lda, ldb, ldc, epi, nullptr, 1, status};
  return out_dtype == TSP_DTYPE_BF16 ? launch<__nv_bfloat16, false>(p, stream) : launch<float, false>(p, stream);
}

// h[m,n] (bf16, optional) = A[m,k] * B[n,k]^T, act[m,n] (bf16) = gelu(h + bias[n]) of the rounded h: a linear layer and its
// activation in one pass.  n a multiple of 64, bias 16-byte aligned.  B200: 12608 x 3072 x 768 with
// both outputs 71 us against 54 + 34 for product and activation, 16384 rows without h 79 against 65 + 43.
int tsp_gemm_bf16_tn_gelu_2cta(const void* a, const void* b, void* h, void* act, const float* bias, int m, int n, int k,
                               int lda, int ldb, int ldc, int* status, cudaStream_t stream) {
  if (m <= 0 || n <= 0 || k <= 0) return 0;
  if ((lda % 8) || (ldb % 8) || (k % 8) || n % 64 != 0 || bias == nullptr || act == nullptr) return -3;
  if (((uintptr_t)a | (uintptr_t)b | (uintptr_t)h | (uintptr_t)act | (uintptr_t)bias) & 15) return -2;
  const Args p = {{a, nullptr, nullptr}, 1, b, {h, act, nullptr}, 2, bias, m, n, k, lda, ldb, ldc, h != nullptr ? 1 : 0,
                  nullptr, 1, status};
  return launch<__nv_bfloat16, false, kGelu>(p, stream);
}

// [C0 | C1 | C2] = A[m,k] * B[n,k]^T (+ bias[n]), bf16: one product whose n columns go to n_dst matrices of n / n_dst
// columns each (a multiple of 64), all with row pitch ldc.  3 x 768 columns of 12608 rows: 49 us, B200,
// against 64 for three products.
int tsp_gemm_bf16_tn_2cta_split(const void* a, const void* b, void* const* c, int n_dst, const float* bias, int m, int n,
                                int k, int lda, int ldb, int ldc, int* status, cudaStream_t stream) {
  if (m <= 0 || n <= 0 || k <= 0) return 0;
  if (n_dst < 1 || n_dst > kMaxCDst || n % n_dst != 0 || (n / n_dst) % 64 != 0) return -3;
  if ((lda % 8) || (ldb % 8) || (k % 8)) return -3;
  if (((uintptr_t)a | (uintptr_t)b) & 15) return -2;
  Args p = {{a, nullptr, nullptr}, 1, b, {c[0], nullptr, nullptr}, n_dst, bias, m, n, k, lda, ldb, ldc,
            bias != nullptr ? 1 : 0, nullptr, 1, status};
  for (int i = 0; i < n_dst; ++i) p.c[i] = c[i];
  return launch<__nv_bfloat16, false>(p, stream);
}

// C[m,n] (bf16) = [A0 | A1 | A2] B with B [k, n] row-major: the gradient of a linear layer's input (A = dY, B = W), or of
// n_src layers that share it (A_i = dY_i, B = their weights stacked).  A_i [m, k / n_src] with row pitch lda; k / n_src a
// multiple of 64 when n_src > 1.
int tsp_gemm_bf16_nn_2cta(const void* const* a, int n_src, const void* b, void* c, int m, int n, int k, int lda, int ldb,
                          int ldc, int* status, cudaStream_t stream) {
  if (m <= 0 || n <= 0 || k <= 0) return 0;
  if (n_src < 1 || n_src > kMaxASrc || k % n_src != 0 || (n_src > 1 && (k / n_src) % BK != 0)) return -3;
  if ((lda % 8) || (ldb % 8)) return -3;
  Args p = {{a[0], nullptr, nullptr}, n_src, b, {c, nullptr, nullptr}, 1, nullptr, m, n, k, lda, ldb, ldc, 0, nullptr, 1, status};
  uintptr_t bits = (uintptr_t)b;
  for (int i = 0; i < n_src; ++i) { p.a[i] = a[i]; bits |= (uintptr_t)a[i]; }
  if (bits & 15) return -2;
  return launch<__nv_bfloat16, false, kNN>(p, stream);
}

// C[m,n] (fp32) += [A0 | A1 | A2]^T B with A_i [k, m / n_src], B [k, n]: the gradient of a linear layer's weight (A = dY,
// B = X), or of the stacked weights of n_src layers that share their input.  m / n_src a multiple of 64 when n_src > 1; C
// 16-byte aligned with a row pitch that is a multiple of 4.
int tsp_gemm_bf16_wgrad_2cta(const void* const* a, int n_src, const void* b, float* c, int m, int n, int k, int lda, int ldb,
                             int ldc, int* status, cudaStream_t stream) {
  if (m <= 0 || n <= 0 || k <= 0) return 0;
  if (n_src < 1 || n_src > kMaxASrc || m % n_src != 0 || (n_src > 1 && (m / n_src) % 64 != 0)) return -3;
  if ((lda % 8) || (ldb % 8)) return -3;
  Args p = {{a[0], nullptr, nullptr}, n_src, b, {c, nullptr, nullptr}, 1, nullptr, m, n, k, lda, ldb, ldc, 0, nullptr, 1, status};
  uintptr_t bits = (uintptr_t)b;
  for (int i = 0; i < n_src; ++i) { p.a[i] = a[i]; bits |= (uintptr_t)a[i]; }
  if (bits & 15) return -2;
  return launch<float, false, kRed>(p, stream);
}

// C (bf16) = A B^T as above, plus per-column statistics of the rounded result for a BatchNorm that follows:
// col_sums [segs][2n] fp32 (zeroed by the caller) receives, for each of the `segs` consecutive groups of
// m / segs rows, the column sums and the column sums of squares.  m / segs must be a multiple of 128; C must be
// 16-byte aligned with a row pitch that is a multiple of 16 bytes.
int tsp_gemm_bf16_tn_2cta_stats(const void* a, const void* b, void* c, int m, int n, int k, int lda, int ldb, int ldc,
                                float* col_sums, int segs, int* status, cudaStream_t stream) {
  if (m <= 0 || n <= 0 || k <= 0) return 0;
  if ((lda % 8) || (ldb % 8) || (k % 8) || segs < 1 || m % segs != 0 || (m / segs) % 128 != 0) return -3;
  if (((uintptr_t)a | (uintptr_t)b) & 15) return -2;
  const Args p = {{a, nullptr, nullptr}, 1, b, {c, nullptr, nullptr}, 1, nullptr, m, n, k, lda, ldb, ldc, 0, col_sums, m / segs,
                  status};
  return launch<__nv_bfloat16, true>(p, stream);
}

}  // extern "C"

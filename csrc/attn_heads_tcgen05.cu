// Attention forward softmax(Q K^T * scale + mask) V for heads of 64, without a gradient (teacher and momentum encoders), with
// an optional boolean mask over the keys: the ViT and BERT blocks of `benchmarks/moco-v3/vits.py` (timm's Attention) and
// `benchmarks/distilbert/bert.py` (HF BertSelfAttention), there two batched products, a softmax and an additive mask.
//
// Persistent, one CTA per SM; an item is 256 queries of one head.  The two tiles of 128 queries take turns: while one's
// scores are in the softmax, the tensor core works on the other's.  The floor are the exponentials, 128 x 128 per tile of queries
// and keys at 16 a clock; what is seen is some twice that, the latency of the way score product - softmax - value product.
// [32, 12, 512, 64] with a padding mask: 58 us (the library 110, most of it for the mask).
//   warp 0      keys and values of 128 keys at a time by TMA, shared by both tiles; the mask as four words of bits per tile;
//               tiles of keys that are all switched off are left out (their probabilities are exact zeros);
//   warps 1, 2  one thread each, one tile of queries each: S = Q K^T (128 x 128 x 64, both from shared memory) and O += P V
//               (A = P from tensor memory); with one thread for both tiles 74 us where two take 70;
//   warps 4-7, 8-11  softmax of the first and second tile, thread = query: P goes back to tensor memory as bf16, never through
//               shared memory; O is rescaled only when a row's maximum has grown by more than 2^8 since the last time (O and
//               the row sum carry the same factor until the division at the end).  The output leaves by TMA through the memory
//               of the item's queries (stored by the threads: 70 us where this takes 58).
// A batch entry whose keys are all switched off attends to all of them, as it does in the library.  Keys and values that are off are not
// read where a whole tile of them is, so that an infinite or NaN one there has no part in anything.  Tensor memory: S 2 x 128 columns, P 2 x 64, O 2 x 64.
// Every mbarrier wait is bounded; a wait that runs out sets *status and all roles leave their loops.
#include <cuda.h>
#include <math.h>

#include "common.cuh"
#include "tcgen05.cuh"
#include "tspipe_kernels.h"

namespace {

constexpr int kTile = 128, kDim = 64;
constexpr int kStages = 4;
constexpr int kTileBytes = kTile * kDim * 2;                    // 128 rows of Q, K or V
constexpr int kSmemBytes = 4 * kTileBytes + kStages * 2 * kTileBytes + 1024 + 512;
constexpr int kThreads = 128 + 256;
constexpr int kMaxKeys = 32 * kTile;
constexpr uint64_t kWaitNs = 2000000000ull;
constexpr float kLog2e = 1.4426950408889634f;
constexpr float kSlackLog2 = 8.f;                               // growth of a maximum that is left in P and O
constexpr uint32_t kColS = 0, kColP = 256, kColO = 384;

struct TileInfo {
  uint32_t keys[4];              // bit per key: takes part
  uint32_t last;                 // of its item
};

__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
      "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
        "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]),
        "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]),
        "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t* r) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr)
               : "memory");
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t* r) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
               ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
               : "memory");
}
__device__ __forceinline__ void tma_store_4d(const CUtensorMap* map, const void* smem_src, int y, int z, int w) {
  asm volatile("cp.async.bulk.tensor.4d.global.shared::cta.bulk_group [%0, {%2, %3, %4, %5}], [%1];" ::"l"(map),
               "r"(tc5::smem_u32(smem_src)), "r"(0), "r"(y), "r"(z), "r"(w)
               : "memory");
  asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}
// A from tensor memory: lane = row, one column = two bf16 neighbours along K
__device__ __forceinline__ void umma_bf16_ta(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc,
                                             uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}

__global__ void __launch_bounds__(kThreads, 1)
attn_heads_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                  const __grid_constant__ CUtensorMap tmap_v, const __grid_constant__ CUtensorMap tmap_o,
                  const uint8_t* __restrict__ mask, int64_t mask_stride, int nq, int nk, int heads, int items, float scale,
                  int* __restrict__ status) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* q_s = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);      // [2 items][2 tiles]
  uint8_t* kv_s = q_s + 4 * kTileBytes;                                            // [kStages][K, V]
  uint64_t* bars = (uint64_t*)(kv_s + kStages * 2 * kTileBytes);
  uint64_t* q_full = bars;                     // [2]
  uint64_t* q_empty = bars + 2;                // [2] softmax -> producer (8 arrivals): the item's output has left the memory of Q
  uint64_t* s_full = bars + 4;                 // [2] per tile: MMA -> softmax
  uint64_t* s_empty = bars + 6;                // [2] softmax -> MMA (4 arrivals): the scores are in registers
  uint64_t* p_full = bars + 8;                 // [2] softmax -> MMA (4 arrivals)
  uint64_t* o_done = bars + 10;                // [2] MMA -> softmax: P has been read, O holds it
  uint64_t* o_empty = bars + 12;               // [2] softmax -> MMA (4 arrivals): O of an item is in registers
  uint64_t* kv_full = bars + 14;               // [kStages]
  uint64_t* kv_empty = kv_full + kStages;      // [kStages] softmax -> producer (8 arrivals), once O holds a tile's product
  uint32_t* tmem_slot = (uint32_t*)(kv_empty + kStages);
  TileInfo* info = (TileInfo*)(tmem_slot + 2);                                     // [kStages]

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int pairs = (nq + 2 * kTile - 1) / (2 * kTile), n_tiles = (nk + kTile - 1) / kTile;
  if (threadIdx.x == 0) {
    for (int i = 0; i < 2; ++i) {
      tc5::mbar_init(q_full + i, 1);
      tc5::mbar_init(q_empty + i, 8);
      tc5::mbar_init(s_full + i, 1);
      tc5::mbar_init(s_empty + i, 4);
      tc5::mbar_init(p_full + i, 4);
      tc5::mbar_init(o_done + i, 1);
      tc5::mbar_init(o_empty + i, 4);
    }
    for (int i = 0; i < kStages; ++i) { tc5::mbar_init(kv_full + i, 1); tc5::mbar_init(kv_empty + i, 8); }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&tmap_q) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&tmap_k) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&tmap_v) : "memory");
  }
  if (warp == 3) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc5::smem_u32(tmem_slot)),
                 "r"(512u)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = *tmem_slot;

  auto arrived = [&](uint64_t* bar, uint32_t parity, int code) -> bool {       // polled, the same for the warp
    return __all_sync(0xffffffffu, tc5::mbar_wait(bar, parity, status, code, kWaitNs)) != 0;
  };
  if (warp == 0) {
    // ---------------- producer ----------------
    uint32_t g = 0, idx = 0;                   // tiles of keys, items
    bool ok = true;
    for (int item = blockIdx.x; item < items && ok; item += gridDim.x, ++idx) {
      const int bh = item / pairs, q0 = (item - bh * pairs) * 2 * kTile, head = bh % heads, bat = bh / heads;
      const uint8_t* mrow = mask != nullptr ? mask + bat * mask_stride : nullptr;
      // this lane's four keys of tile j, one bit each
      auto nibble = [&](int j) -> uint32_t {
        uint32_t v = 0;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int key = j * kTile + 4 * lane + i;
          if (key < nk && (mrow == nullptr || mrow[key] != 0)) v |= 1u << i;
        }
        return v;
      };
      uint32_t active = 0;
      for (int j = 0; j < n_tiles; ++j)
        if (mrow == nullptr || __any_sync(0xffffffffu, nibble(j) != 0)) active |= 1u << j;
      if (active == 0) {                       // no key at all: as without a mask, which is what the library's kernel gives from two keys on
        mrow = nullptr;
        active = n_tiles == 32 ? 0xffffffffu : (1u << n_tiles) - 1;
      }
      if (idx >= 2) ok = tc5::mbar_wait_warp(q_empty + (idx & 1), ((idx >> 1) - 1) & 1, status, 1, kWaitNs, lane);
      if (!ok) break;
      if (lane == 0) {
        tc5::mbar_expect_tx(q_full + (idx & 1), 2 * kTileBytes);
        uint8_t* dst = q_s + (idx & 1) * 2 * kTileBytes;
        for (int i = 0; i < 2; ++i)            // rows past the last query read as zeros
          tc5::tma_load_4d(dst + i * kTileBytes, &tmap_q, q_full + (idx & 1), 0, q0 + i * kTile, head, bat);
      }
      for (int j = 0; j < n_tiles; ++j) {
        if (!(active >> j & 1)) continue;
        const uint32_t s = g % kStages, round = g / kStages;
        uint32_t word = nibble(j) << (4 * (lane & 7));
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) word |= __shfl_xor_sync(0xffffffffu, word, o);
        if (round > 0 && !tc5::mbar_wait_warp(kv_empty + s, (round - 1) & 1, status, 1, kWaitNs, lane)) { ok = false; break; }
        if ((lane & 7) == 0) info[s].keys[lane >> 3] = word;
        if (lane == 0) info[s].last = (active >> j) == 1u ? 1u : 0u;
        __syncwarp();
        if (lane == 0) {
          uint8_t* dst = kv_s + s * 2 * kTileBytes;
          tc5::mbar_expect_tx(kv_full + s, 2 * kTileBytes);
          tc5::tma_load_4d(dst, &tmap_k, kv_full + s, 0, j * kTile, head, bat);
          tc5::tma_load_4d(dst + kTileBytes, &tmap_v, kv_full + s, 0, j * kTile, head, bat);
        }
        ++g;
      }
    }
  } else if (warp == 1 || warp == 2) {
    // ---------------- MMA issuer of one tile of queries ----------------
    {
      const int w = warp - 1;
      const bool issuer = tc5::elect_one();
      constexpr uint32_t idesc_s = tc5::make_idesc(kTile, kTile, false, false);
      constexpr uint32_t idesc_o = tc5::make_idesc(kTile, kDim, false, true);
      const uint64_t q_desc = tc5::desc_k_major(tc5::smem_u32(q_s)), k_desc = tc5::desc_k_major(tc5::smem_u32(kv_s));
      const uint64_t v_desc = tc5::desc_mn_major(tc5::smem_u32(kv_s) + kTileBytes, kTileBytes);
      uint32_t g = 0, idx = 0, n_s = 0;                // tiles of keys whose O is under way, items, score products
      bool ok = true, last = false;
      auto issue_s = [&]() -> bool {                   // of the next tile of keys
        const uint32_t stage = n_s % kStages;
        if (!arrived(kv_full + stage, (n_s / kStages) & 1, 2)) return false;
        if (n_s > 0 && !arrived(s_empty + w, (n_s - 1) & 1, 4)) return false;
        last = ((volatile TileInfo*)info)[stage].last != 0;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint64_t q = q_desc + (uint64_t)(((idx & 1) * 2 + w) * (kTileBytes >> 4));
        const uint64_t k = k_desc + (uint64_t)(stage * (2 * kTileBytes >> 4));
        if (issuer) {
#pragma unroll
          for (int kk = 0; kk < kDim / 16; ++kk)
            tc5::umma_bf16(tmem_base + kColS + w * kTile, q + (uint64_t)(2 * kk), k + (uint64_t)(2 * kk), idesc_s, kk > 0 ? 1u : 0u);
          tc5::umma_commit(s_full + w);
        }
        __syncwarp();
        ++n_s;
        return true;
      };
      for (int item = blockIdx.x; item < items && ok; item += gridDim.x, ++idx) {
        ok = arrived(q_full + (idx & 1), (idx >> 1) & 1, 2) && issue_s();
        for (bool first = true; ok; first = false, ++g) {
          const bool more = !last;
          ok = (!more || issue_s()) && arrived(p_full + w, g & 1, 5) &&
               (!first || idx == 0 || arrived(o_empty + w, (idx - 1) & 1, 6));
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint64_t v = v_desc + (uint64_t)(g % kStages * (2 * kTileBytes >> 4));
          if (issuer) {
#pragma unroll
            for (int ks = 0; ks < kTile / 16; ++ks)    // 16 keys: 8 columns of P, 16 rows of V
              umma_bf16_ta(tmem_base + kColO + w * kDim, tmem_base + kColP + w * (kTile / 2) + ks * 8, v + (uint64_t)(ks * 128),
                           idesc_o, !first || ks > 0 ? 1u : 0u);
            tc5::umma_commit(o_done + w);
          }
          __syncwarp();
          if (!more) { ++g; break; }
        }
      }
    }
  } else if (warp >= 4) {
    // ---------------- softmax + epilogue: thread = query ----------------
    const int w = (warp - 4) >> 2, quarter = warp & 3;
    const uint32_t lane_addr = tmem_base + ((uint32_t)(quarter * 32) << 16);
    const float sc2 = scale * kLog2e;
    uint32_t g = 0, idx = 0;
    bool ok = true;
    for (int item = blockIdx.x; item < items && ok; item += gridDim.x, ++idx) {
      float m_run = -INFINITY, l_run = 0.f;            // the maximum that P and O refer to, log2 domain
      for (bool first = true; ok; first = false) {
        const uint32_t s = g % kStages;
        ok = arrived(kv_full + s, (g / kStages) & 1, 3) &&
             arrived(s_full + w, g & 1, 3);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        float x[kTile];
#pragma unroll
        for (int c0 = 0; c0 < kTile; c0 += 32)
          tc5::tmem_ld_32x32_issue(lane_addr + kColS + w * kTile + c0, reinterpret_cast<uint32_t*>(x) + c0);
        uint32_t keys[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) keys[i] = ((volatile TileInfo*)info)[s].keys[i];
        const bool last = ((volatile TileInfo*)info)[s].last != 0;
        tc5::tmem_ld_wait();
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) tc5::mbar_arrive(s_empty + w);
        if ((keys[0] & keys[1] & keys[2] & keys[3]) != 0xffffffffu) {
#pragma unroll
          for (int c = 0; c < kTile; ++c) x[c] = keys[c >> 5] >> (c & 31) & 1 ? x[c] : -INFINITY;
        }
        float top[4] = {x[0], x[1], x[2], x[3]};
#pragma unroll
        for (int c = 4; c < kTile; ++c) top[c & 3] = fmaxf(top[c & 3], x[c]);
        const float mx = fmaxf(fmaxf(top[0], top[1]), fmaxf(top[2], top[3])) * sc2;
        float alpha = 1.f;
        if (mx > m_run + kSlackLog2 || m_run == -INFINITY) {
          const float m_new = fmaxf(m_run, mx);
          alpha = m_run == -INFINITY ? 0.f : ex2(m_run - m_new);
          m_run = m_new;
        }
        const float m_use = m_run == -INFINITY ? 0.f : m_run;
        if (!first) {                                  // the product before has read P, and O holds it
          ok = arrived(o_done + w, (g - 1) & 1, 7);
          if (!ok) break;
          if (lane == 0) tc5::mbar_arrive(kv_empty + (g - 1) % kStages);
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          if (!__all_sync(0xffffffffu, alpha == 1.f)) {
#pragma unroll 1
            for (int c0 = 0; c0 < kDim; c0 += 8) {     // (rare; few registers beside the scores)
              uint32_t o[8];
              tmem_ld8(lane_addr + kColO + w * kDim + c0, o);
              tc5::tmem_ld_wait();
#pragma unroll
              for (int e = 0; e < 8; ++e) o[e] = __float_as_uint(__uint_as_float(o[e]) * alpha);
              tmem_st8(lane_addr + kColO + w * kDim + c0, o);
            }
          }
        }
        float sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int c0 = 0; c0 < kTile; c0 += 64) {
          uint32_t p[32];
#pragma unroll
          for (int c = 0; c < 64; c += 2) {
            const float a = ex2(fmaf(x[c0 + c], sc2, -m_use)), b = ex2(fmaf(x[c0 + c + 1], sc2, -m_use));
            sum[c & 2] += a;
            sum[(c & 2) + 1] += b;
            p[c / 2] = tc5::pack_bf16x2(a, b);
          }
          tmem_st32(lane_addr + kColP + w * (kTile / 2) + c0 / 2, p);
        }
        l_run = l_run * alpha + ((sum[0] + sum[1]) + (sum[2] + sum[3]));
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) {
          tc5::mbar_arrive(p_full + w);
          if (first && idx > 0) {                      // the output of the item before has been read by now
            asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
            tc5::mbar_arrive(q_empty + ((idx - 1) & 1));
          }
        }
        __syncwarp();
        ++g;
        if (!last) continue;
        // ---------------- O / l ----------------
        ok = arrived(o_done + w, (g - 1) & 1, 8);
        if (!ok) break;
        if (lane == 0) tc5::mbar_arrive(kv_empty + (g - 1) % kStages);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        uint32_t o[kDim];
        tc5::tmem_ld_32x32_issue(lane_addr + kColO + w * kDim, o);
        tc5::tmem_ld_32x32_issue(lane_addr + kColO + w * kDim + 32, o + 32);
        tc5::tmem_ld_wait();
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) tc5::mbar_arrive(o_empty + w);
        // the queries' tile is not read any more: the output leaves through it
        const int bh = item / pairs, row0 = (item - bh * pairs) * 2 * kTile + w * kTile + quarter * 32;
        const float inv = l_run == 0.f ? 0.f : 1.f / l_run;
        uint8_t* block = q_s + ((idx & 1) * 2 + w) * kTileBytes + quarter * 32 * 128;
#pragma unroll
        for (int q = 0; q < kDim / 8; ++q) {
          uint32_t v[4];
#pragma unroll
          for (int e = 0; e < 4; ++e)
            v[e] = tc5::pack_bf16x2(__uint_as_float(o[8 * q + 2 * e]) * inv, __uint_as_float(o[8 * q + 2 * e + 1]) * inv);
          *reinterpret_cast<uint4*>(block + lane * 128 + ((q ^ (lane & 7)) << 4)) = make_uint4(v[0], v[1], v[2], v[3]);
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0 && row0 < nq) tma_store_4d(&tmap_o, block, row0, bh % heads, bh / heads);      // rows past nq are clipped
        break;
      }
    }
  }
  if (warp >= 4 && lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  if (*((volatile int*)status) != 0) tc5::drain_in_flight();
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 3) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
  }
}

bool head_map(CUtensorMap* map, const void* p, int n, int heads, int batch, const int64_t* strides, int rows = kTile) {
  const uint64_t dims[4] = {kDim, (uint64_t)n, (uint64_t)heads, (uint64_t)batch};
  const uint64_t bytes[4] = {2, (uint64_t)strides[0] * 2, (uint64_t)strides[1] * 2, (uint64_t)strides[2] * 2};
  const uint32_t box[4] = {kDim, (uint32_t)rows, 1, 1};
  return tc5::make_bf16_map(map, p, 4, dims, bytes, box);
}

}  // namespace

extern "C" {

// out[b, i, h, :] (bf16, contiguous) = softmax over the keys j with mask[b, j] != 0 (all of them without a mask) of
// scale * q[b, h, i, :] k[b, h, j, :]^T, times v[b, h, j, :]; heads of 64.  Strides are {row, head, batch} in elements,
// multiples of 8; bases 16-byte aligned; at most 4096 keys.  mask: bytes, keys contiguous, `mask_stride` bytes per batch.
// `status`: one zeroed int in device memory; non-zero afterwards = a bounded wait ran out and out is not valid.
int tsp_attn_heads_fwd(const void* q, const void* k, const void* v, const uint8_t* mask, int64_t mask_stride, void* out,
                       int batch, int heads, int nq, int nk, const int64_t* q_strides, const int64_t* k_strides,
                       const int64_t* v_strides, float scale, int* status, cudaStream_t stream) {
  if (batch <= 0 || heads <= 0 || nq <= 0) return 0;
  if (nk < 1 || nk > kMaxKeys || !(scale > 0.f)) return -3;
  if ((((uintptr_t)q | (uintptr_t)k | (uintptr_t)v | (uintptr_t)out) & 15) != 0) return -2;
  for (const int64_t* st : {q_strides, k_strides, v_strides})
    for (int i = 0; i < 3; ++i)
      if (st[i] <= 0 || st[i] % 8 != 0) return -3;
  const int64_t items = (int64_t)batch * heads * ((nq + 2 * kTile - 1) / (2 * kTile));
  if (items > 0x7fffffff) return -3;
  CUtensorMap tq, tk, tv, to;
  const int64_t o_strides[3] = {(int64_t)heads * kDim, kDim, (int64_t)nq * heads * kDim};
  if (!head_map(&tq, q, nq, heads, batch, q_strides) || !head_map(&tk, k, nk, heads, batch, k_strides) ||
      !head_map(&tv, v, nk, heads, batch, v_strides) || !head_map(&to, out, nq, heads, batch, o_strides, 32))
    return -6;
  int usable = 0;
  cudaError_t e = tsp::usable_sms(usable);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(attn_heads_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes);
  if (e != cudaSuccess) return (int)e;
  attn_heads_kernel<<<items < usable ? (int)items : usable, kThreads, kSmemBytes, stream>>>(
      tq, tk, tv, to, mask, mask_stride, nq, nk, heads, (int)items, scale, status);
  return TSP_LAUNCH_CHECK();
}

}  // extern "C"

// Persistent tcgen05 GEMM for large problems (bf16 and single-pass TF32).
//
// Pairs of CTAs (one per SM, clusters of two) walk a list of 256 x 256 output tiles with tcgen05.mma.cta_group::2:
// each CTA fetches 128 rows of A and 128 of the 256 rows of B, the tensor cores of both read B from both shared
// memories, and each CTA holds 128 rows of the accumulator.  Compared with the one-tile-per-CTA kernel of gemm_tc.cuh:
//   * per 512 cycles of tensor work a CTA fetches and reads 32 KB of operands (64 KB at 128 x 128, 48 KB at 128 x 256);
//     what bounds the product in a running step is the power limit, and operand traffic is what is left to save;
//   * the accumulator is double-buffered in tensor memory (2 x 256 columns =
//     all 512): the epilogue warps drain tile i while the MMA warp already
//     accumulates tile i+1, and the TMA ring never drains between tiles;
//   * set-up (barriers, TMEM allocation, descriptor prefetch) is paid once per
//     SM instead of once per tile.
// Tiles are visited in groups of kGroupM row-tiles x all column-tiles so that
// the pairs running at the same time share operand slabs in L2.  The schedule
// is dynamic: the producer thread of the even CTA (the leader) draws the next work item from a counter in
// global memory and hands it to the other roles of both CTAs through a small ring in
// shared memory, so a pair that starts late (SMs held by a kernel of another
// stream, e.g. a collective) simply finds less work left instead of delaying
// a fixed share of the tiles.  The pair that draws the last ticket of the
// launch (n_items + pairs - 1) resets the counter for the next launch.
//
// The tiles of the last, partial wave may be split in K (weight gradients: fp32 C, no fused epilogue): a work item is
// then one K range of one tile, added into C.
//
// Roles (12 warps): warp 0 TMA producer (the bytes of both CTAs are counted on the leader's barrier), warp 1 TMEM
// owner and, in the leader, MMA issuer for the pair (its commits reach the barriers of both CTAs), warps 4-11 epilogue in two groups (warp w drains TMEM lanes 32(w%4)..+31;
// group 0 takes the even 128-byte column chunks of a tile, group 1 the odd ones).  C leaves and the ReLU mask comes in
// boxes of 32 rows x 128 bytes through the tensor maps, two per warp in turn, the mask's box becoming the output's in
// place (whole lines instead of 64-byte pieces of 32 lines per instruction); fp32 sums (beta = 1, K ranges) as
// reductions on the way.  The register path stays for other beta and for unaligned C.  Every mbarrier
// wait is bounded (see mbar_wait); after a failed wait all roles stop and the
// CTA still frees its tensor memory.
// Measured (graph replay; 128 x 256 tiles of single CTAs before): 8192x4096x4096 bias + ReLU 188 us (201), masked 197 (215),
// 8192x4096x1000 masked 70 (80), 4096x4096x8192 weight gradient 197 (233), 8192x1000x4096 56 (62), TF32 4096^3 238 (272).
#pragma once

#include "gemm_tc.cuh"

namespace zg {
namespace tc {

constexpr int kPBM = 256, kPBN = 256;  // tile of a pair
constexpr int kGroupM = 8;     // row-tiles per scheduling group
constexpr int kThreadsPersistent = 384;
constexpr int kEpiWarps = kThreadsPersistent / 32 - 4;
constexpr int kSchedDepth = 4;                  // work items in flight between the roles
constexpr uint32_t kNoTile = 0xFFFFFFFFu;       // end of work
constexpr uint32_t kNoSplit = 0xFFFFFFFFu;      // the whole k range

template <int MODE>
struct PersistentSmem {
  using MT = ModeTraits<MODE>;
  static constexpr int kABytes = kBM * kSlabBytes;    // 16 KB
  static constexpr int kBBytes = kPBN / 2 * kSlabBytes;  // 16 KB: this CTA's half
  static constexpr int kStageBytes = kABytes + kBBytes;
  static constexpr int kStages = 5;
  static constexpr int kBoxes = 2 * kEpiWarps;        // two output boxes of 32 rows x 128 bytes per epilogue warp
  static constexpr int kTotal = kStages * kStageBytes + kBoxes * 4096 + 1024 /*alignment slack*/ + 512 /*barriers*/;
};

// Address of the same shared-memory object in CTA `rank` of the pair
__device__ __forceinline__ uint32_t map_rank(const void* p, uint32_t rank) { return map_rank(smem_u32(p), rank); }
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// Bounded like mbar_wait, with the arrivals of the other CTA's threads ordered before what follows
__device__ __forceinline__ bool mbar_wait_cluster(uint64_t* bar, uint32_t parity, volatile int* failed) {
  for (uint32_t it = 0; it < kSpinLimit; ++it) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    if (ok) return true;
    if (it > 64) {
      if (*failed) return false;
      __nanosleep(40);
    }
  }
  *failed = 1;
  return false;
}
// Load into this CTA's shared memory whose bytes are counted on a barrier of either CTA of the pair
__device__ __forceinline__ void tma_load_3d_pair(void* smem_dst, const CUtensorMap* map, uint32_t bar, int x, int y, int z) {
  asm volatile(
      "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(map), "r"(bar), "r"(x), "r"(y), "r"(z)
      : "memory");
}
template <bool BF16>
__device__ __forceinline__ void umma_pair(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  if constexpr (BF16) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
  } else {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::tf32 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
  }
}
// The barrier at this place in both CTAs arrives once all previously issued MMAs of this thread are done
__device__ __forceinline__ void umma_commit_pair(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
               ::"r"(smem_u32(bar)), "h"((uint16_t)3)
               : "memory");
}
// All but the latest N bulk groups of this thread have read their shared-memory source
template <int N>
__device__ __forceinline__ void bulk_wait_read() {
  asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(N) : "memory");
}

struct TileCoord { uint32_t m, n, batch, split; };

// tile index -> (row-tile, column-tile, batch); groups of kGroupM row-tiles, row-tile fastest inside a group
__device__ __forceinline__ TileCoord tile_coord(uint32_t t, uint32_t tiles_m, uint32_t tiles_n, uint32_t whole, uint32_t splits) {
  TileCoord c;
  c.split = kNoSplit;
  if (t >= whole) {
    c.split = (t - whole) % splits;  // the K ranges of a tile are neighbours in the list: they run at the same time
    t = whole + (t - whole) / splits;
  }
  const uint32_t per_batch = tiles_m * tiles_n;
  c.batch = t / per_batch;
  t -= c.batch * per_batch;
  const uint32_t group_sz = kGroupM * tiles_n;
  const uint32_t g = t / group_sz, in_g = t - g * group_sz;
  const uint32_t m0 = g * kGroupM;
  const uint32_t gm = (tiles_m - m0) < (uint32_t)kGroupM ? (tiles_m - m0) : (uint32_t)kGroupM;
  c.n = in_g / gm;
  c.m = m0 + (in_g - c.n * gm);
  return c;
}

template <bool A_KMAJOR, bool B_KMAJOR, int MODE>
__global__ void __launch_bounds__(kThreadsPersistent, 1)
gemm_tc_persistent_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                          const __grid_constant__ CUtensorMap tmC, const __grid_constant__ CUtensorMap tmM, const Params p,
                          const uint32_t tiles_m, const uint32_t tiles_n, const uint32_t n_tiles, unsigned* sched_counter) {
  static_assert(MODE == kBF16 || MODE == kTF32, "the persistent kernel has no operand-split warps");
  using MT = ModeTraits<MODE>;
  using SL = PersistentSmem<MODE>;
  constexpr int S = SL::kStages;
  constexpr int BN = kPBN;
  constexpr uint32_t kIdesc = make_idesc(MT::kBf16, !A_KMAJOR, !B_KMAJOR, BN) + ((uint32_t)((kPBM - kBM) >> 4) << 24);
  constexpr uint32_t kTmemCols = 512;  // two 256-column accumulators

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint8_t* boxes = smem + S * SL::kStageBytes;
  uint64_t* bars = reinterpret_cast<uint64_t*>(boxes + SL::kBoxes * 4096);
  uint64_t* full = bars;                 // [S] TMA bytes of both CTAs landed (the leader's)
  uint64_t* empty = bars + S;            // [S] MMAs that read the stage retired
  uint64_t* acc_full = bars + 2 * S;     // [2] accumulator complete
  uint64_t* acc_empty = bars + 2 * S + 2;  // [2] accumulator drained by the epilogues of both CTAs (the leader's)
  uint64_t* sched_full = bars + 2 * S + 4;                 // [kSchedDepth] work item published
  uint64_t* sched_empty = bars + 2 * S + 4 + kSchedDepth;  // [kSchedDepth] read by the leader's MMA warp, the other
                                                           // CTA's producer and every epilogue warp (the leader's)
  uint64_t* mask_full = sched_empty + kSchedDepth;         // [kBoxes] mask box landed
  __shared__ uint32_t sched_tile[kSchedDepth];
  __shared__ uint32_t tmem_base_slot;
  __shared__ volatile int failed;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = blockIdx.x & 1;  // in the pair; 0 leads
  // k-slabs of K range `split` (p.k_per_split is a multiple of the slab depth)
  auto slabs_of = [&](uint32_t split) -> int {
    if (split == kNoSplit) return (int)((p.k + MT::kBK - 1) / MT::kBK);
    const uint32_t kb = split * p.k_per_split;
    if (kb >= p.k) return 0;
    const uint32_t ke = (kb + p.k_per_split < p.k) ? kb + p.k_per_split : p.k;
    return (int)((ke - kb + MT::kBK - 1) / MT::kBK);
  };

  if (threadIdx.x == 0) {
    failed = 0;
    for (int s = 0; s < S; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&acc_full[b], 1);
      mbar_init(&acc_empty[b], 2 * kEpiWarps);
    }
    for (int j = 0; j < kSchedDepth; ++j) {
      mbar_init(&sched_full[j], 1);
      mbar_init(&sched_empty[j], 2 + 2 * kEpiWarps);
    }
    for (int b = 0; b < SL::kBoxes; ++b) mbar_init(&mask_full[b], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    prefetch_tmap(&tmA);
    prefetch_tmap(&tmB);
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_slot)), "r"(kTmemCols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync();  // the other CTA's barriers and tensor memory are there
  tc_fence_after();
  const uint32_t tmem_base = tmem_base_slot;
  pdl_sync();  // everything above overlaps the previous kernel's tail

  if (warp == 0) {
    // ------------------------------------------------------------ producer
    if (lane == 0) {
      uint32_t it = 0;  // k-slabs issued so far (ring position)
      bool ok = true;
      for (uint32_t i = 0; ok; ++i) {
        const int j = (int)(i % kSchedDepth);
        uint32_t t;
        if (rank == 0) {
          if (i >= (uint32_t)kSchedDepth && !mbar_wait_cluster(&sched_empty[j], ((i / kSchedDepth) & 1) ^ 1, &failed)) break;
          t = atomicAdd(sched_counter, 1u);
          if (t == n_tiles + gridDim.x / 2 - 1) atomicExch(sched_counter, 0u);  // the last draw of the launch
          if (t >= n_tiles) t = kNoTile;
          sched_tile[j] = t;
          mbar_arrive(&sched_full[j]);
          asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(map_rank(&sched_tile[j], 1)), "r"(t) : "memory");
          mbar_arrive_cluster(map_rank(&sched_full[j], 1));
        } else {
          if (!mbar_wait_cluster(&sched_full[j], (i / kSchedDepth) & 1, &failed)) break;
          t = sched_tile[j];
          mbar_arrive_cluster(map_rank(&sched_empty[j], 0));
        }
        if (t == kNoTile) break;
        const TileCoord tc = tile_coord(t, tiles_m, tiles_n, p.whole_tiles, p.splits);
        const int za = (int)(tc.batch % p.nA), zb = (int)(tc.batch % p.nB);
        const int KT = slabs_of(tc.split);
        for (int kt = 0; kt < KT; ++kt, ++it) {
          const int s = (int)(it % S);
          if (it >= (uint32_t)S && !mbar_wait(&empty[s], ((it / S) & 1) ^ 1, &failed)) { ok = false; break; }
          uint8_t* a_dst = smem + s * SL::kStageBytes;
          uint8_t* b_dst = a_dst + SL::kABytes;
          if (rank == 0) mbar_expect_tx(&full[s], 2 * SL::kStageBytes);
          const uint32_t bar = map_rank(&full[s], 0);
          const int k0 = (int)(tc.split == kNoSplit ? 0u : tc.split * p.k_per_split) + kt * MT::kBK;
          const int m0 = (int)(tc.m * kPBM + rank * kBM), n0 = (int)(tc.n * BN + rank * (BN / 2));
          if (A_KMAJOR) {
            tma_load_3d_pair(a_dst, &tmA, bar, k0, m0, za);
          } else {
#pragma unroll
            for (int j = 0; j < kBM / MT::kAtomMN; ++j)
              tma_load_3d_pair(a_dst + j * MT::kBK * kSlabBytes, &tmA, bar, m0 + j * MT::kAtomMN, k0, za);
          }
          if (B_KMAJOR) {
            tma_load_3d_pair(b_dst, &tmB, bar, k0, n0, zb);
          } else {
#pragma unroll
            for (int j = 0; j < BN / 2 / MT::kAtomMN; ++j)
              tma_load_3d_pair(b_dst + j * MT::kBK * kSlabBytes, &tmB, bar, n0 + j * MT::kAtomMN, k0, zb);
          }
        }
      }
    }
  } else if (warp == 1) {
    // ---------------------------------------------------------- MMA issuer
    // The whole warp walks the loops (waits and descriptor arithmetic stay
    // warp-uniform), one elected lane issues the MMAs and the commits; the
    // barrier of the next ring position is tested before this slab's MMAs go out.
    if (rank == 0) {
      uint32_t it = 0, tcount = 0;
      bool ok = true, have = false;
      for (; ok; ++tcount) {
        const int j = (int)(tcount % kSchedDepth);
        bool got = mbar_wait(&sched_full[j], (tcount / kSchedDepth) & 1, &failed);
        if (!__all_sync(0xffffffffu, got)) break;
        const uint32_t t = sched_tile[j];
        __syncwarp();
        if (lane == 0) mbar_arrive(&sched_empty[j]);
        if (t == kNoTile) break;
        const uint32_t buf = tcount & 1;
        if (tcount >= 2) {
          got = mbar_wait_cluster(&acc_empty[buf], ((tcount >> 1) & 1) ^ 1, &failed);
          if (!__all_sync(0xffffffffu, got)) break;
        }
        tc_fence_after();
        const uint32_t tmem_d = tmem_base + buf * BN;
        const int KT = slabs_of(tile_coord(t, tiles_m, tiles_n, p.whole_tiles, p.splits).split);
        for (int kt = 0; kt < KT; ++kt, ++it) {
          const int s = (int)(it % S);
          if (!have) {
            got = mbar_wait(&full[s], (it / S) & 1, &failed);
            if (!__all_sync(0xffffffffu, got)) { ok = false; break; }
          }
          const uint32_t it1 = it + 1;
          const bool next_seen = mbar_test(&full[it1 % S], (it1 / S) & 1);
          tc_fence_after();
          const uint32_t a_s = smem_u32(smem + s * SL::kStageBytes), b_s = a_s + SL::kABytes;
          constexpr uint32_t a_step = (A_KMAJOR ? 32u : (uint32_t)(MT::kUmmaK * kSlabBytes)) >> 4;
          constexpr uint32_t b_step = (B_KMAJOR ? 32u : (uint32_t)(MT::kUmmaK * kSlabBytes)) >> 4;
          constexpr uint32_t a_lbo = A_KMAJOR ? 16u : (uint32_t)(MT::kBK * kSlabBytes);
          constexpr uint32_t b_lbo = B_KMAJOR ? 16u : (uint32_t)(MT::kBK * kSlabBytes);
          constexpr uint32_t a_lay = (!A_KMAJOR && !MT::kBf16) ? 1u : 2u, b_lay = (!B_KMAJOR && !MT::kBf16) ? 1u : 2u;
          constexpr uint32_t a_h32 = desc_hi32(a_lay == 1u ? 512u : 1024u, a_lay), b_h32 = desc_hi32(b_lay == 1u ? 512u : 1024u, b_lay);
          const uint32_t da0 = desc_lo32(a_s, a_lbo), db0 = desc_lo32(b_s, b_lbo);
          if (elect_one()) {
#pragma unroll
            for (int kk = 0; kk < MT::kBK / MT::kUmmaK; ++kk)
              umma_pair<MT::kBf16>(tmem_d, desc_pack(da0 + kk * a_step, a_h32), desc_pack(db0 + kk * b_step, b_h32), kIdesc,
                              (kt > 0 || kk > 0) ? 1u : 0u);
            umma_commit_pair(&empty[s]);
          }
          have = __all_sync(0xffffffffu, next_seen);
        }
        if (ok && elect_one()) umma_commit_pair(&acc_full[buf]);
      }
    }
  } else if (warp >= 4) {
    // ------------------------------------------------------------ epilogue
    const int q = warp & 3, group = (warp - 4) >> 2;
    uint8_t* stg = boxes + (warp - 4) * 8192;
    uint64_t* mbar = mask_full + (warp - 4) * 2;
    const bool out16 = p.Cb != nullptr, masked = p.epilogue == ZG_EPI_RELU_MASK, tma = p.tma_epilogue != 0;
    const bool has_bias = p.epilogue == ZG_EPI_BIAS || p.epilogue == ZG_EPI_BIAS_RELU;
    const int width = tma && out16 ? 64 : 32;  // columns of a chunk: 128 bytes of C
    uint32_t box = 0;                          // output boxes of this warp so far
    uint32_t tcount = 0;
    for (;; ++tcount) {
      const int j = (int)(tcount % kSchedDepth);
      if (!mbar_wait_cluster(&sched_full[j], (tcount / kSchedDepth) & 1, &failed)) break;
      const uint32_t t = sched_tile[j];
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(map_rank(&sched_empty[j], 0));
      if (t == kNoTile) break;
      const uint32_t buf = tcount & 1;
      const TileCoord tc = tile_coord(t, tiles_m, tiles_n, p.whole_tiles, p.splits);
      const int KT = slabs_of(tc.split);
      const uint32_t row0 = tc.m * kPBM + rank * kBM + q * 32, row = row0 + lane;
      const uint32_t n_left = p.n - tc.n * BN;  // columns of C from this tile on
      int chunks = (int)((min(n_left, (uint32_t)BN) + width - 1) / width);
      if (row0 >= p.m) chunks = 0;
      auto fetch_mask = [&](int c, uint32_t b) {  // lane 0; the stores out of box b have been read
        mbar_expect_tx(&mbar[b & 1], 4096);
        tma_load_3d(stg + (b & 1) * 4096, &tmM, &mbar[b & 1], (int)(tc.n * BN) + c * width, (int)row0, (int)tc.batch);
      };
      if (tma && masked && group < chunks && lane == 0) {
        bulk_wait_read<0>();
        fetch_mask(group, box);
      }
      if (!mbar_wait(&acc_full[buf], (tcount >> 1) & 1, &failed)) break;
      tc_fence_after();
      const uint64_t c_off = (uint64_t)tc.batch * p.c_batch_stride + (uint64_t)row * p.ldc;
      const bool row_ok = row < p.m;
      const uint32_t acc = tmem_base + buf * BN + ((uint32_t)(q * 32) << 16);
      bool ok = true;
#pragma unroll 1
      for (int c = group; c < chunks; c += 2) {
        uint8_t* rowp = stg + (box & 1) * 4096 + lane * 128;
        if (tma) {
          if (lane == 0) {
            if (!masked) bulk_wait_read<1>();
            else if (c + 2 < chunks) {
              bulk_wait_read<0>();
              fetch_mask(c + 2, box + 1);
            }
          }
          __syncwarp();
        }
#pragma unroll 1
        for (int half = 0; half < width / 32; ++half) {
          const uint32_t col0 = tc.n * BN + c * width + half * 32;
          if (col0 >= p.n) break;
          uint32_t r[32];
          if (KT > 0) {
            tmem_ld32(acc + (uint32_t)(c * width + half * 32), r);
            tmem_ld_wait();
          } else {
#pragma unroll
            for (int j = 0; j < 32; ++j) r[j] = 0u;
          }
          if (!tma) {
            epilogue_chunk(p, r, row_ok, c_off + col0, col0, lane);
            continue;
          }
          float v[32];
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = p.alpha * __uint_as_float(r[j]);
          if (has_bias) {
            if (col0 + 32 <= p.n) {
#pragma unroll
              for (int j = 0; j < 8; ++j) {
                const float4 bv = __ldg(reinterpret_cast<const float4*>(p.bias + col0) + j);
                v[4 * j] += bv.x; v[4 * j + 1] += bv.y; v[4 * j + 2] += bv.z; v[4 * j + 3] += bv.w;
              }
            } else {
#pragma unroll
              for (int j = 0; j < 32; ++j)
                if (col0 + j < p.n) v[j] += __ldg(p.bias + col0 + j);
            }
            if (p.epilogue == ZG_EPI_BIAS_RELU) {
#pragma unroll
              for (int j = 0; j < 32; ++j) v[j] = v[j] > 0.f ? v[j] : 0.f;
            }
          } else if (masked && half == 0) {
            ok = mbar_wait(&mbar[box & 1], (box >> 1) & 1, &failed);
          }
          if (out16) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              uint4* at = reinterpret_cast<uint4*>(rowp + (((half * 4 + j) ^ (lane & 7)) << 4));
              if (masked) {
                const uint4 u = *at;
                const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                  const float2 f = __bfloat1622float2(h[i]);
                  if (f.x <= 0.f) v[8 * j + 2 * i] = 0.f;
                  if (f.y <= 0.f) v[8 * j + 2 * i + 1] = 0.f;
                }
              }
              uint4 u;
              __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&u);
#pragma unroll
              for (int i = 0; i < 4; ++i) h[i] = __floats2bfloat162_rn(v[8 * j + 2 * i], v[8 * j + 2 * i + 1]);
              *at = u;
            }
          } else {
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              float4* at = reinterpret_cast<float4*>(rowp + ((j ^ (lane & 7)) << 4));
              if (masked) {
                const float4 u = *at;
                if (u.x <= 0.f) v[4 * j] = 0.f;
                if (u.y <= 0.f) v[4 * j + 1] = 0.f;
                if (u.z <= 0.f) v[4 * j + 2] = 0.f;
                if (u.w <= 0.f) v[4 * j + 3] = 0.f;
              }
              *at = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
            }
          }
          if (p.colsum) {
            if (!row_ok) {
#pragma unroll
              for (int j = 0; j < 32; ++j) v[j] = 0.f;
            }
            colsum_chunk(p, v, col0, lane);
          }
        }
        if (!tma) continue;
        fence_async_smem();  // generic-proxy writes -> visible to the TMA unit
        __syncwarp();
        if (lane == 0) {
          const int x = (int)(tc.n * BN) + c * width;
          if (p.tma_epilogue == 2 || (p.tma_epilogue == 3 && tc.split != kNoSplit)) tma_reduce_add_box(&tmC, stg + (box & 1) * 4096, x, (int)row0, (int)tc.batch);
          else tma_store_box(&tmC, stg + (box & 1) * 4096, x, (int)row0, (int)tc.batch);
          bulk_commit_group();
        }
        ++box;
      }
      if (!__all_sync(0xffffffffu, ok)) break;
      // all tcgen05.ld of this warp have completed (wait::ld): hand the accumulator back
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(map_rank(&acc_empty[buf], 0));
    }
    if (lane == 0) bulk_wait_read<0>();
  }

  // ---------------------------------------------------------------- teardown
  if (failed) asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(map_rank((const void*)&failed, rank ^ 1)), "r"(1) : "memory");
  tc_fence_before();
  __syncthreads();
  if (failed) outstay_own_work();
  cluster_sync();  // nobody's MMAs, loads or arrivals are under way any more
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kTmemCols) : "memory");
  }
  if (threadIdx.x == 0 && failed && p.error_flag) *p.error_flag = 1;
}

}  // namespace tc
}  // namespace zg

// tcgen05 / TMEM / TMA GEMM for sm_100a.
//
//   C[b] = epilogue(alpha * op(A[b % nA]) * op(B[b % nB]) + beta * C[b])
//
// One CTA computes one 128 x BN tile of C (optionally one K-split of it).
// Roles inside the CTA (8 warps):
//   warp 0      TMA producer: cp.async.bulk.tensor loads of the A and B
//               k-slabs into a ring of shared-memory stages (128-byte swizzle)
//   warp 1      MMA issuer: the whole warp walks the k loop (so waits and
//               descriptor arithmetic stay warp-uniform; a loop run by a single
//               lane measured 55 cycles per tcgen05.mma issued against 20 this
//               way), one elected lane issues tcgen05.mma with the accumulator
//               in tensor memory; also owns the TMEM allocation
//   warps 2-11  FP32X3 mode only (the other modes have 8 warps): for every fp32
//               operand slab form the remainder lo = x - tf32(x).  The MMA reads
//               only the top 19 bits of an fp32 word (measured: results do not
//               change when the low 13 bits are cleared first), so the fetched
//               word itself serves as "hi" and Ahi*Bhi + Alo*Bhi + Ahi*Blo
//               recovers fp32-level accuracy.  Hi and lo of A go to tensor memory
//               (thread = row), lo of B to a second buffer of the stage.  Warps
//               4-7 and 8-11 take the A slabs in turn, warps 2-3 split (most of)
//               B, each fetching its part of its next slab before it hands the
//               current one over; one mbarrier arrival per warp.  With one set of
//               A warps the serial chain of a slab (wait, split, tcgen05.st, wait)
//               bounded the loop: 4096^3 650 -> 635 us, 128x784x8192 12.7 -> 12.3
//   warps 12-19 DIRECT instances only: element-wise copies of operands whose rows no
//               TMA box can address (1000x501x1000 with 501-float rows: 16 us
//               against 66 on the FFMA path, 4096x1023x1023 80 against 385)
//   kBF16Sums   (bf16 operands, fp32 C): an accumulator takes the products of two or four instructions only, two accumulators in
//               turn, and warps 4-7 add them up in registers, rounding to nearest; the tensor core's own sums
//               truncate at every instruction (1895x1340x2310 2.4e-6 off in the 2-norm, 1.3e-7 like this)
//   warps 4-7   read the accumulator (tcgen05.ld: warp q reads TMEM lanes
//               32q..32q+31, one row per thread); then either staged boxes go to
//               the TMA unit, or the whole tile is staged in shared memory and
//               all warps apply alpha / beta / bias / ReLU / mask with lanes along
//               the rows of C, so that unaligned rows are coalesced as well.
//               Split K forms clusters of up to 8 CTAs that sum their staged tiles
//               through distributed shared memory in rank order: 2000x256x1000 +
//               bias + ReLU 30 -> 14 us (before: partial sums added into a
//               pre-scaled C by atomics, the last CTA of a tile re-reading it)
//
// Operand layouts.  A row-major matrix whose contiguous dimension is K is a
// "K-major" UMMA operand; one whose contiguous dimension is M (or N) is
// "MN-major".  Both are fetched by TMA into the canonical 128-byte-swizzled
// layouts that the shared-memory matrix descriptors name:
//   K-major  : slab = rows x 128 bytes of K; 8-row groups are 1024 bytes apart
//              (SBO); the k-th MMA inside the slab starts 32 bytes further
//   MN-major : slab = column blocks of 128 bytes of M/N; inside a block the
//              k rows are 128 bytes apart, swizzle-row groups are SBO apart,
//              column blocks BK*128 bytes apart (LBO).  16-bit types use the
//              plain 128-byte swizzle (8-row groups, SBO 1024); 32-bit types
//              must use the 128-byte swizzle with 32-byte atoms (4-row groups,
//              SBO 512) -- the only MN-major layout tcgen05 accepts for tf32
//
// Every wait on an mbarrier is bounded: when the limit is reached the CTA
// raises a flag in global memory, stops issuing work, and still releases its
// tensor memory before it returns.
#pragma once

#include <cuda.h>
#include <cuda_bf16.h>
#include <cstdint>

#include "common.cuh"

namespace zg {
namespace tc {

constexpr int kBM = 128;
constexpr int kThreadsTc = 256;
constexpr int kSplitThreads = kThreadsTc - 64;  // warps 2-7
constexpr int kSlabBytes = 128;          // bytes of the contiguous dimension per smem row
constexpr uint32_t kSpinLimit = 1u << 24;  // polls per wait before giving up

enum Mode { kTF32 = 0, kFP32X3 = 1, kBF16 = 2, kBF16Sums = 3 };  // kBF16Sums: bf16 operands, fp32 sums that round (below)

struct Params {
  float* C;             // fp32 output (or nullptr when Cb is used)
  __nv_bfloat16* Cb;    // bf16 output
  const float* bias;    // [n] or nullptr
  float* colsum;        // [n] or nullptr: column sums of the stored values are ADDED here (fp32 atomics)
  const float* mask;    // fp32 mask source with C's layout (when C is fp32)
  const __nv_bfloat16* maskb;
  uint64_t c_batch_stride;  // elements
  uint32_t m, n, k;
  uint32_t ldc;
  uint32_t nA, nB;      // operand batch counts (index wraps)
  uint32_t tiles_n;     // column tiles
  uint32_t splits;      // K splits (gridDim.x = column tiles * splits)
  uint32_t whole_tiles; // persistent kernel: the first tiles of the list, which are not split
  uint32_t k_per_split; // multiple of BK
  float alpha, beta;
  int epilogue;
  int vec_ok;           // C (and mask, bias) rows allow 16-byte accesses at every 32-column boundary
  int* error_flag;      // set to 1 when a bounded wait ran out
  // Epilogue through the C tensor map (fp32 C with 16-byte-aligned rows): each epilogue warp stages its
  // 32 rows of a 32-column chunk in shared memory (128-byte swizzle) and one lane hands the box to the
  // TMA unit -- 1: plain store (no split-K, beta == 0, epilogue NONE / BIAS / BIAS_RELU, no column
  // sums), 2: reduce-add into C (split-K partial products; C pre-scaled by beta).  Whole 128-byte
  // lines leave the SM instead of 16-byte pieces of 32 different lines per instruction, and boxes that
  // hang over the edge of C are clipped by the unit.  3 (persistent kernel): whole tiles are stored, K ranges added into
  // tiles that were cleared.  0: register path below.
  int tma_epilogue;
  // Split K over the CTAs of a cluster: every CTA stages its partial tile in shared memory, rank r sums rows r,
  // r + splits, ... of all of them through distributed shared memory in rank order and applies the epilogue.
  int cluster;
  int swap;  // the tile is C transposed: its rows are C's columns (short C: the long dimension fills the 128 rows)
  // Operands whose rows no TMA box can address (base or row stride not a multiple of 16 bytes) come through
  // element-wise cp.async of loader warps into the same swizzled slabs (DIRECT instances only).
  int a_direct, b_direct;
  const float* a_src;
  const float* b_src;
  uint64_t a_ld, b_ld, a_batch, b_batch;  // elements
};

// ------------------------------------------------------------------ PTX
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Non-blocking test of a phase (try_wait may suspend the thread for a while when the phase is
// still open; a look-ahead must not)
__device__ __forceinline__ bool mbar_test(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Bounded wait.  Returns false (and raises *failed) when the limit is hit or
// another role already failed.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, volatile int* failed) {
  for (uint32_t it = 0; it < kSpinLimit; ++it) {
    if (mbar_try_wait(bar, parity)) return true;
    if (it > 64) {
      if (*failed) return false;
      __nanosleep(40);
    }
  }
  *failed = 1;
  return false;
}

__device__ __forceinline__ void tma_load_3d(void* smem_dst, const CUtensorMap* map, uint64_t* bar, int x, int y, int z) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(map), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z)
      : "memory");
}
__device__ __forceinline__ void prefetch_tmap(const CUtensorMap* map) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(map) : "memory");
}

__device__ __forceinline__ void tmem_alloc(uint32_t* dst_smem, uint32_t cols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst_smem)), "r"(cols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t cols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// D[tmem] (+)= A[smem desc] * B[smem desc]
template <bool BF16>
__device__ __forceinline__ void umma(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  if constexpr (BF16) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
  } else {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
  }
}
// One lane of a converged warp (the same lane every time for the full mask)
__device__ __forceinline__ bool elect_one() {
  uint32_t pred;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(pred));
  return pred != 0;
}
// mbarrier arrives once all previously issued MMAs of this thread are done
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// 32 lanes x 32 consecutive fp32 columns: thread t gets row (lane base + t)
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
        "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]),
        "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
        "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
// 32 lanes x 32 consecutive 32-bit columns: thread t writes row (lane base + t)
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
      "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
        "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]),
        "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]),
        "r"(r[30]), "r"(r[31])
      : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// D[tmem] (+)= A[tmem] * B[smem desc], tf32: A is read from tensor memory (row m in lane m, one k element per column)
__device__ __forceinline__ void umma_tmem_a(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// Shared-memory matrix descriptor (tcgen05): start address, leading-dimension
// byte offset and stride byte offset in 16-byte units, descriptor version 1,
// 128-byte swizzle.
// `layout`: 2 = 128-byte swizzle, 1 = 128-byte swizzle with 32-byte atoms.
__device__ __forceinline__ uint64_t make_desc(uint32_t smem_addr, uint32_t lbo_bytes, uint32_t sbo_bytes, uint32_t layout) {
  uint64_t d = 0;
  d |= (uint64_t)((smem_addr >> 4) & 0x3FFF);
  d |= (uint64_t)((lbo_bytes >> 4) & 0x3FFF) << 16;
  d |= (uint64_t)((sbo_bytes >> 4) & 0x3FFF) << 32;
  d |= (uint64_t)1 << 46;  // version (Blackwell)
  d |= (uint64_t)layout << 61;
  return d;
}

// The same descriptor as two 32-bit halves: the upper half is a compile-time
// constant of the layout, the lower half is (address >> 4) | (LBO >> 4) << 16,
// so stepping to the next MMA inside a slab is ONE integer add on the lower
// half (the MMA-issuing thread is a single in-order thread; this keeps its
// work per tcgen05.mma at a few instructions).
__host__ __device__ constexpr uint32_t desc_hi32(uint32_t sbo_bytes, uint32_t layout) {
  return ((sbo_bytes >> 4) & 0x3FFFu) | (1u << 14) | (layout << 29);
}
__device__ __forceinline__ uint32_t desc_lo32(uint32_t smem_addr, uint32_t lbo_bytes) {
  return ((smem_addr >> 4) & 0x3FFFu) | (((lbo_bytes >> 4) & 0x3FFFu) << 16);
}
__device__ __forceinline__ uint64_t desc_pack(uint32_t lo, uint32_t hi) {
  uint64_t d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "r"(lo), "r"(hi));
  return d;
}

// Instruction descriptor: fp32 accumulate, A/B format (tf32 = 2, bf16 = 1),
// operand majors, N >> 3, M >> 4.
__host__ __device__ constexpr uint32_t make_idesc(bool bf16, bool a_mn_major, bool b_mn_major, int N) {
  return (1u << 4) | ((bf16 ? 1u : 2u) << 7) | ((bf16 ? 1u : 2u) << 10) | ((a_mn_major ? 1u : 0u) << 15) |
         ((b_mn_major ? 1u : 0u) << 16) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(kBM >> 4) << 24);
}

// shared -> global through a tensor map, tracked by the issuing thread's bulk async-group
__device__ __forceinline__ void tma_store_box(const CUtensorMap* map, const void* smem_src, int x, int y, int z) {
  asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%2, %3, %4}], [%1];"
               ::"l"(map), "r"(smem_u32(smem_src)), "r"(x), "r"(y), "r"(z)
               : "memory");
}
__device__ __forceinline__ void tma_reduce_add_box(const CUtensorMap* map, const void* smem_src, int x, int y, int z) {
  asm volatile("cp.reduce.async.bulk.tensor.3d.global.shared::cta.add.tile.bulk_group [%0, {%2, %3, %4}], [%1];"
               ::"l"(map), "r"(smem_u32(smem_src)), "r"(x), "r"(y), "r"(z)
               : "memory");
}
__device__ __forceinline__ void bulk_commit_group() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
// until the bulk operations of this thread have READ their shared-memory source (their global writes are
// complete when the grid completes, which is what a dependent kernel waits for)
__device__ __forceinline__ void bulk_wait_group_read() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }

template <int MODE>
struct ModeTraits {
  static constexpr bool kBf16 = (MODE == kBF16 || MODE == kBF16Sums);
  static constexpr int kElem = kBf16 ? 2 : 4;
  static constexpr int kBK = kSlabBytes / kElem;       // elements of K per stage: 32 (fp32) / 64 (bf16)
  static constexpr int kUmmaK = 32 / kElem;            // K per MMA: 8 (tf32) / 16 (bf16)
  static constexpr int kAtomMN = kSlabBytes / kElem;   // M/N elements per 128-byte column block
};

// Column sums of this warp's 32 x 32 block without shared memory: five exchange rounds, each halving the columns a lane
// still carries (a lane keeps the half selected by its own bit); lane j ends with column j.
__device__ __forceinline__ void colsum_chunk(const Params& p, float (&v)[32], uint32_t col0, int lane) {
#pragma unroll
  for (int off = 16; off >= 1; off >>= 1) {
    const bool upper = (lane & off) != 0;
#pragma unroll
    for (int j = 0; j < off; ++j) {
      const float send = upper ? v[j] : v[j + off];
      const float keep = upper ? v[j + off] : v[j];
      v[j] = keep + __shfl_xor_sync(0xffffffffu, send, off);
    }
  }
  if (col0 + lane < p.n) atomicAdd(p.colsum + col0 + lane, v[0]);
}

// Epilogue of one 32-column chunk of one accumulator row (registers r, raw
// fp32 bits): alpha/beta/bias/ReLU/mask, the store (or the split-K reduction
// into C), and the optional column sums.  `o` = element offset of (row, col0)
// in C; warp-collective when p.colsum is set.
__device__ __forceinline__ void epilogue_chunk(const Params& p, const uint32_t (&r)[32], bool row_ok, uint64_t o, uint32_t col0, int lane) {
  if (!row_ok && !p.colsum) return;
  const bool need_c = p.beta != 0.f, need_m = p.epilogue == ZG_EPI_RELU_MASK;
  const bool has_bias = p.epilogue == ZG_EPI_BIAS || p.epilogue == ZG_EPI_BIAS_RELU;
  float v[32];
#pragma unroll
  for (int j = 0; j < 32; ++j) v[j] = p.alpha * __uint_as_float(r[j]);
  const bool full = p.vec_ok && (col0 + 32 <= p.n);
  if (!row_ok) {
#pragma unroll
    for (int j = 0; j < 32; ++j) v[j] = 0.f;
  } else if (full) {
    if (p.splits > 1) {
      // C was pre-scaled by beta on the host side; no fused epilogue with split-K
#pragma unroll
      for (int j = 0; j < 32; j += 4)
        asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p.C + o + j), "f"(v[j]), "f"(v[j + 1]), "f"(v[j + 2]), "f"(v[j + 3]) : "memory");
      return;
    }
    if (p.C) {  // fp32 C / mask
      if (need_c) {
        float4 cv[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) cv[j] = *reinterpret_cast<const float4*>(p.C + o + 4 * j);
#pragma unroll
        for (int j = 0; j < 8; ++j) { v[4 * j] += p.beta * cv[j].x; v[4 * j + 1] += p.beta * cv[j].y; v[4 * j + 2] += p.beta * cv[j].z; v[4 * j + 3] += p.beta * cv[j].w; }
      }
      if (has_bias) {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float4 bv = __ldg(reinterpret_cast<const float4*>(p.bias + col0) + j);
          v[4 * j] += bv.x; v[4 * j + 1] += bv.y; v[4 * j + 2] += bv.z; v[4 * j + 3] += bv.w;
        }
        if (p.epilogue == ZG_EPI_BIAS_RELU) {
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = v[j] > 0.f ? v[j] : 0.f;
        }
      } else if (need_m) {
        float4 mv[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) mv[j] = *reinterpret_cast<const float4*>(p.mask + o + 4 * j);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          if (mv[j].x <= 0.f) v[4 * j] = 0.f;
          if (mv[j].y <= 0.f) v[4 * j + 1] = 0.f;
          if (mv[j].z <= 0.f) v[4 * j + 2] = 0.f;
          if (mv[j].w <= 0.f) v[4 * j + 3] = 0.f;
        }
      }
#pragma unroll
      for (int j = 0; j < 8; ++j)
        *reinterpret_cast<float4*>(p.C + o + 4 * j) = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
    } else {  // bf16 C / mask: 32 values = 64 bytes = 4 x 16-byte accesses
      if (need_c) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const uint4 u = *reinterpret_cast<const uint4*>(p.Cb + o + 8 * j);
          const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
          for (int t = 0; t < 4; ++t) { const float2 f = __bfloat1622float2(h[t]); v[8 * j + 2 * t] += p.beta * f.x; v[8 * j + 2 * t + 1] += p.beta * f.y; }
        }
      }
      if (has_bias) {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float4 bv = __ldg(reinterpret_cast<const float4*>(p.bias + col0) + j);
          v[4 * j] += bv.x; v[4 * j + 1] += bv.y; v[4 * j + 2] += bv.z; v[4 * j + 3] += bv.w;
        }
        if (p.epilogue == ZG_EPI_BIAS_RELU) {
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = v[j] > 0.f ? v[j] : 0.f;
        }
      } else if (need_m) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const uint4 u = *reinterpret_cast<const uint4*>(p.maskb + o + 8 * j);
          const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
          for (int t = 0; t < 4; ++t) {
            const float2 f = __bfloat1622float2(h[t]);
            if (f.x <= 0.f) v[8 * j + 2 * t] = 0.f;
            if (f.y <= 0.f) v[8 * j + 2 * t + 1] = 0.f;
          }
        }
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        uint4 u;
        __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&u);
#pragma unroll
        for (int t = 0; t < 4; ++t) h[t] = __floats2bfloat162_rn(v[8 * j + 2 * t], v[8 * j + 2 * t + 1]);
        *reinterpret_cast<uint4*>(p.Cb + o + 8 * j) = u;
      }
    }
  } else {
    // ragged edge or unaligned C: element-wise with a column bound
    const uint32_t ncol = (p.n - col0) < 32u ? (p.n - col0) : 32u;
#pragma unroll
    for (uint32_t j = 0; j < 32; ++j) {
      if (j < ncol) {
        float x = v[j];
        if (p.splits > 1) { atomicAdd(p.C + o + j, x); continue; }
        if (need_c) x += p.beta * (p.C ? p.C[o + j] : __bfloat162float(p.Cb[o + j]));
        if (has_bias) { x += p.bias[col0 + j]; if (p.epilogue == ZG_EPI_BIAS_RELU) x = x > 0.f ? x : 0.f; }
        else if (need_m) { if ((p.mask ? p.mask[o + j] : __bfloat162float(p.maskb[o + j])) <= 0.f) x = 0.f; }
        if (p.C) p.C[o + j] = x;
        else p.Cb[o + j] = __float2bfloat16_rn(x);
        v[j] = x;
      } else {
        v[j] = 0.f;
      }
    }
  }
  if (p.colsum) colsum_chunk(p, v, col0, lane);
}

// 32 columns of one accumulator row; with two accumulators `apart` columns from one another, their sum
template <bool TWO>
__device__ __forceinline__ void load_accumulator(uint32_t taddr, uint32_t apart, uint32_t (&r)[32]) {
  tmem_ld32(taddr, r);
  if constexpr (TWO) {
    uint32_t small[32];
    tmem_ld32(taddr + apart, small);
    tmem_ld_wait();
#pragma unroll
    for (int j = 0; j < 32; ++j) r[j] = __float_as_uint(__uint_as_float(r[j]) + __uint_as_float(small[j]));
  } else {
    tmem_ld_wait();
  }
}

// One row of an fp32 A slab (32 k values of row `row` of the 128-row tile) from its shared-memory stage.
// K-major: the row is 128 contiguous bytes whose 16-byte chunks sit at position c ^ (row % 8).
// MN-major: the stage holds four column blocks of 32 rows; a block is 32 k-rows of 128 bytes (32
// consecutive rows of A) whose 32-byte atoms sit at position atom ^ (k % 4); the read transposes.
template <bool A_KMAJOR>
__device__ __forceinline__ void load_a_row(const uint8_t* a_stage, int row, float4 (&v)[8]) {
  if constexpr (A_KMAJOR) {
    const uint8_t* rp = a_stage + row * kSlabBytes;
#pragma unroll
    for (int c = 0; c < 8; ++c) v[c] = *reinterpret_cast<const float4*>(rp + ((c ^ (row & 7)) << 4));
  } else {
    const uint8_t* bp = a_stage + (row >> 5) * (32 * kSlabBytes) + ((row & 7) << 2);
    const int atom = (row >> 3) & 3;
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      v[c].x = *reinterpret_cast<const float*>(bp + (4 * c + 0) * kSlabBytes + ((atom ^ 0) << 5));
      v[c].y = *reinterpret_cast<const float*>(bp + (4 * c + 1) * kSlabBytes + ((atom ^ 1) << 5));
      v[c].z = *reinterpret_cast<const float*>(bp + (4 * c + 2) * kSlabBytes + ((atom ^ 2) << 5));
      v[c].w = *reinterpret_cast<const float*>(bp + (4 * c + 3) * kSlabBytes + ((atom ^ 3) << 5));
    }
  }
}

constexpr int kLoadWarps = 8;
// One slab (ROWS rows x 32 k) of an fp32 operand into its swizzled place by 256 threads, 4 bytes per copy, lanes along
// the contiguous dimension of the source.  The four warps' issue rate bounds it (a predicate and a pointer select per
// copy made a 128x128 slab pair 2300 cycles, twice what its MMAs take), so a whole slab of whole k is an add and a copy
// each.  Rows past the end of a K-major source repeat the last one (what they give lies outside C), elsewhere they are
// zeroed: lanes that copy from one address are served one by one (2708x7x2708: 28 us against 13).  Past k the slab is zero.
template <int ROWS, bool KMAJOR>
__device__ __forceinline__ void direct_slab(uint8_t* dst, const float* src, uint64_t ld, uint32_t row0, uint32_t rows, uint32_t k0, uint32_t k) {
  const int w = (threadIdx.x >> 5) & 7, lane = threadIdx.x & 31;
  const uint32_t base = smem_u32(dst);
  auto copy = [&](uint32_t to, const float* from) { asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(to), "l"(from) : "memory"); };
  auto copy_if = [&](uint32_t to, const float* from, bool ok) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(to), "l"(ok ? from : src), "r"(ok ? 4 : 0) : "memory");
  };
  const bool whole_k = k0 + 32 <= k;
  if constexpr (KMAJOR) {
    const uint32_t d = base + w * kSlabBytes + (((lane >> 2) ^ w) << 4) + ((lane & 3) << 2);
    const uint32_t first = row0 + w < rows ? row0 + w : rows - 1;
    const float* s = src + (uint64_t)first * ld + k0 + lane;
    const uint64_t step = 8 * ld;
    auto to = [&](int i) { return d + i * (8 * kSlabBytes); };
    if (whole_k && row0 + ROWS <= rows) {
#pragma unroll
      for (int i = 0; i < ROWS / 8; ++i) { copy(to(i), s); s += step; }
    } else {
      const bool k_ok = k0 + lane < k;
#pragma unroll 8
      for (int i = 0; i < ROWS / 8; ++i) {
        copy_if(to(i), s, k_ok);
        if (row0 + w + 8 * (i + 1) < rows) s += step;
      }
    }
  } else {
    const uint32_t d = base + w * kSlabBytes + (((lane >> 3) ^ (w & 3)) << 5) + ((lane & 7) << 2);
    const float* s = src + (uint64_t)(k0 + w) * ld + row0 + lane;
    const uint64_t step = 8 * ld;
    if (whole_k && row0 + ROWS <= rows) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
#pragma unroll
        for (int b = 0; b < ROWS / 32; ++b) copy(d + b * (32 * kSlabBytes) + i * (8 * kSlabBytes), s + 32 * b);
        s += step;
      }
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const bool k_ok = k0 + w + 8 * i < k;
#pragma unroll
        for (int b = 0; b < ROWS / 32; ++b)
          copy_if(d + b * (32 * kSlabBytes) + i * (8 * kSlabBytes), s + 32 * b, k_ok && row0 + 32 * b + lane < rows);
        s += step;
      }
    }
  }
}

// FP32X3 keeps the hi and lo parts of the A operand in TENSOR
// MEMORY (written by the split warps with tcgen05.st, read by the MMA from
// there): shared memory then holds A once per stage (the fetched slab) and no
// MMA reads it, which takes 64 of the 144 KB per 128x64x32 slab off the
// shared-memory data pipe -- the unit that bounds this mode.
template <int BN, int MODE>
struct SmemLayout {
  static constexpr bool X3 = MODE == kFP32X3;
  using MT = ModeTraits<MODE>;
  static constexpr int kABytes = kBM * kSlabBytes;   // 16 KB
  static constexpr int kBBytes = BN * kSlabBytes;
  static constexpr int kStageBytes = kABytes + (X3 ? 2 : 1) * kBBytes;
  static constexpr int kEpiBytes = 0;
  static constexpr int kBudget = 220 * 1024;
  // FP32X3: a second accumulator behind the first, see the MMA issuer; kBF16Sums: the slabs' products take two in turn
  static constexpr int kAccOne = BN < 32 ? 32 : BN, kAccCols = X3 || MODE == kBF16Sums ? 2 * kAccOne : kAccOne;
  static constexpr int kInPart = BN == 64 ? 2 : 4;  // kBF16Sums: instructions whose products share an accumulator
  static constexpr int kATmemCols = 64;              // per stage: 32 columns hi + 32 columns lo
  static constexpr int kStagesSmem = (kBudget - kEpiBytes - 1024) / kStageBytes;
  static constexpr int kStagesTmem = X3 ? (512 - kAccCols) / kATmemCols : 8;
  static constexpr int kStagesRaw = kStagesSmem < kStagesTmem ? kStagesSmem : kStagesTmem;
  // Even: the two sets of A warps take the slabs in turn, and a set may wait for a slab only if it has waited for the
  // one that filled the same stage before (a parity tells two phases apart, not three).
  static constexpr int kStages = kStagesRaw > 8 ? 8 : kStagesRaw / 2 * 2;
  static constexpr int kTmemNeed = X3 ? kAccCols + kATmemCols * kStages : kAccCols;
  static constexpr int kTmemCols = kTmemNeed <= 32 ? 32 : (kTmemNeed <= 64 ? 64 : (kTmemNeed <= 128 ? 128 : (kTmemNeed <= 256 ? 256 : 512)));
  static constexpr int kTotal = kStages * kStageBytes + kEpiBytes + 1024 /*alignment slack*/ + 256 /*barriers*/;
  // FP32X3: 16-byte words of a B slab per thread of the two B warps / of the four A warps
  // (BN 128: 8 + 4, BN 64: 6 + 1, BN 32: 4 + 0; 64 * kBWordsB + 128 * kBWordsA = BN * 8)
  static constexpr int kBWordsA = BN >= 128 ? 4 : (BN >= 64 ? 1 : 0);
  static constexpr int kBWordsB = (BN * 8 - 128 * kBWordsA) / 64;
  // FP32X3: two sets of four A warps take the slabs in turn
  static constexpr int kThreads = X3 ? 384 : kThreadsTc;  // + kLoadWarps * 32 with direct operands
  static constexpr int kOutPitch = BN + 4;  // floats per row of the staged output tile
  static constexpr int kColRows = (kThreads + kLoadWarps * 32) / (BN / 4);  // partial column sums behind the tile
  static_assert((kBM * kOutPitch + kColRows * BN) * 4 <= kStages * kStageBytes, "the output tile and its column sums are staged in the ring");
};

// One lane's four columns of a row of the staged tile.  VEC: four consecutive columns with 16-byte (fp32) or 8-byte (bf16)
// accesses; else columns `stride` apart, so that the lanes of a warp run along C's row either way.
// What the epilogue needs of C and the mask is requested before the sums are fetched ...
template <bool VEC>
__device__ __forceinline__ void fetch_row4(const Params& p, uint64_t row_off, uint32_t col, uint32_t stride, float (&c)[4], float (&mk)[4]) {
  const bool masked = p.epilogue == ZG_EPI_RELU_MASK;
#pragma unroll
  for (int j = 0; j < 4; ++j) { c[j] = 0.f; mk[j] = 1.f; }
  if constexpr (VEC) {
    const uint64_t o = row_off + col;
    auto get4 = [&](const float* f, const __nv_bfloat16* h, float (&d)[4]) {
      if (f) {
        const float4 x = *reinterpret_cast<const float4*>(f + o);
        d[0] = x.x; d[1] = x.y; d[2] = x.z; d[3] = x.w;
      } else {
        const uint2 u = *reinterpret_cast<const uint2*>(h + o);
        const float2 x = __bfloat1622float2(reinterpret_cast<const __nv_bfloat162*>(&u)[0]), y = __bfloat1622float2(reinterpret_cast<const __nv_bfloat162*>(&u)[1]);
        d[0] = x.x; d[1] = x.y; d[2] = y.x; d[3] = y.y;
      }
    };
    if (p.beta != 0.f) get4(p.C, p.Cb, c);
    if (masked) get4(p.mask, p.maskb, mk);
  } else {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint32_t x = col + j * stride;
      if (x >= p.n) continue;
      if (p.beta != 0.f) c[j] = p.C ? p.C[row_off + x] : __bfloat162float(p.Cb[row_off + x]);
      if (masked) mk[j] = p.mask ? p.mask[row_off + x] : __bfloat162float(p.maskb[row_off + x]);
    }
  }
}
// ... then alpha / beta / bias / ReLU / mask and the store (or the reduction into C)
template <bool VEC>
__device__ __forceinline__ void store_row4(const Params& p, float (&v)[4], uint64_t row_off, uint32_t col, uint32_t stride, const float (&bias)[4],
                                           const float (&c)[4], const float (&mk)[4]) {
  if (p.splits > 1 && !p.cluster) {
    if constexpr (VEC) {
      asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p.C + row_off + col), "f"(p.alpha * v[0]), "f"(p.alpha * v[1]), "f"(p.alpha * v[2]), "f"(p.alpha * v[3]) : "memory");
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (col + j * stride < p.n) atomicAdd(p.C + row_off + col + j * stride, p.alpha * v[j]);
    }
    return;
  }
  const bool relu = p.epilogue == ZG_EPI_BIAS_RELU;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    v[j] = p.alpha * v[j];
    if (p.beta != 0.f) v[j] += p.beta * c[j];
    v[j] += bias[j];
    if (relu) v[j] = v[j] > 0.f ? v[j] : 0.f;
    if (mk[j] <= 0.f) v[j] = 0.f;  // (1 where there is no mask)
  }
  if constexpr (VEC) {
    const uint64_t o = row_off + col;
    if (p.C) {
      *reinterpret_cast<float4*>(p.C + o) = make_float4(v[0], v[1], v[2], v[3]);
    } else {
      uint2 u;
      reinterpret_cast<__nv_bfloat162*>(&u)[0] = __floats2bfloat162_rn(v[0], v[1]);
      reinterpret_cast<__nv_bfloat162*>(&u)[1] = __floats2bfloat162_rn(v[2], v[3]);
      *reinterpret_cast<uint2*>(p.Cb + o) = u;
    }
  } else {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint32_t x = col + j * stride;
      if (x >= p.n) { v[j] = 0.f; continue; }
      if (p.C) p.C[row_off + x] = v[j];
      else p.Cb[row_off + x] = __float2bfloat16_rn(v[j]);
    }
  }
}

// The same for one element (r, c) of a tile that is C transposed
__device__ __forceinline__ float store_swapped(const Params& p, float v, uint64_t o, uint32_t col, float bias) {
  v *= p.alpha;
  if (p.beta != 0.f) v += p.beta * (p.C ? p.C[o] : __bfloat162float(p.Cb[o]));
  v += bias;
  if (p.epilogue == ZG_EPI_BIAS_RELU) v = v > 0.f ? v : 0.f;
  if (p.epilogue == ZG_EPI_RELU_MASK && (p.mask ? p.mask[o] : __bfloat162float(p.maskb[o])) <= 0.f) v = 0.f;
  if (p.C) p.C[o] = v;
  else p.Cb[o] = __float2bfloat16_rn(v);
  return v;
}

__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t map_rank(uint32_t smem_addr, uint32_t rank) {
  uint32_t a;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_addr), "r"(rank));
  return a;
}
__device__ __forceinline__ float4 ld_cluster4(uint32_t a) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ float ld_cluster(uint32_t a) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
  return v;
}

// A staged tile that is C transposed: rows of the tile are columns of C, lanes run along them; a rank takes every
// ranks-th row of C.
template <int BN, int NT>
__device__ __forceinline__ void staged_out_swapped(const Params& p, const float* tile, uint32_t split, uint32_t c0, uint32_t r0, uint64_t batch_off) {
  constexpr int PITCH = BN + 4;
  const uint32_t ranks = p.cluster ? p.splits : 1, rank = p.cluster ? split : 0, r = threadIdx.x % kBM, col = c0 + r;
  if (col >= p.n) return;
  const float bias = (p.epilogue == ZG_EPI_BIAS || p.epilogue == ZG_EPI_BIAS_RELU) ? __ldg(p.bias + col) : 0.f;
  const uint32_t base = smem_u32(tile);
  float cs = 0.f;
#pragma unroll 4
  for (uint32_t c = rank + threadIdx.x / kBM * ranks; c < (uint32_t)BN && r0 + c < p.m; c += NT / kBM * ranks) {
    float v = 0.f;
    const uint32_t at = r * PITCH + c;
    if (ranks == 1) {
      v = tile[at];
    } else {
      float x[8];
#pragma unroll
      for (uint32_t k = 0; k < 8; ++k) x[k] = k < ranks ? ld_cluster(map_rank(base, k) + at * 4) : 0.f;
#pragma unroll
      for (uint32_t k = 0; k < 8; ++k) v += x[k];
    }
    cs += store_swapped(p, v, batch_off + (uint64_t)(r0 + c) * p.ldc + col, col, bias);
  }
  if (p.colsum) atomicAdd(p.colsum + col, cs);
}

// The staged tile (128 x BN floats, pitch BN + 4, all CTAs of a cluster hold partial sums) to C: NT threads, lanes along
// the rows of C, U rows in flight (a row of a lone CTA is a round trip to memory for C and the mask; one of a cluster
// already has a load to every rank in flight, two measured slower).  The column sums of a CTA are
// added up in a fixed order behind the tile.
template <int BN, int NT, bool VEC, int U>
__device__ __forceinline__ void staged_out(const Params& p, float* tile, uint32_t split, uint32_t m0, uint32_t n0, uint64_t batch_off) {
  constexpr int CG = BN / 4, PITCH = BN + 4;
  const uint32_t cg = threadIdx.x % CG, ranks = p.cluster ? p.splits : 1, rank = p.cluster ? split : 0;
  const uint32_t local = VEC ? 4 * cg : cg, stride = VEC ? 1 : CG, col = n0 + local;
  if (col < p.n) {
    float bias[4] = {0.f, 0.f, 0.f, 0.f}, cs[4] = {0.f, 0.f, 0.f, 0.f};
    if (p.epilogue == ZG_EPI_BIAS || p.epilogue == ZG_EPI_BIAS_RELU) {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (col + j * stride < p.n) bias[j] = __ldg(p.bias + col + j * stride);
    }
    const uint32_t base = smem_u32(tile), step = NT / CG * ranks;
    for (uint32_t r0 = rank + threadIdx.x / CG * ranks; r0 < (uint32_t)kBM && m0 + r0 < p.m; r0 += U * step) {
      float v[U][4], c[U][4], mk[U][4];
      bool ok[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const uint32_t r = r0 + u * step;
        ok[u] = r < (uint32_t)kBM && m0 + r < p.m;
        if (ok[u]) fetch_row4<VEC>(p, batch_off + (uint64_t)(m0 + r) * p.ldc, col, stride, c[u], mk[u]);
      }
      if (ranks == 1) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
          if (!ok[u]) continue;
          const float* at = tile + (r0 + u * step) * PITCH + local;
          if constexpr (VEC) {
            const float4 x = *reinterpret_cast<const float4*>(at);
            v[u][0] = x.x; v[u][1] = x.y; v[u][2] = x.z; v[u][3] = x.w;
          } else {
#pragma unroll
            for (int j = 0; j < 4; ++j) v[u][j] = at[j * stride];
          }
        }
      } else {
        // every rank's values are requested before the first is added: one round trip over the cluster network
        float4 x[U][8];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          if (!ok[u]) continue;
          const uint32_t at = ((r0 + u * step) * PITCH + local) * 4;
#pragma unroll
          for (uint32_t k = 0; k < 8; ++k) {
            x[u][k] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (k < ranks) {
              const uint32_t a = map_rank(base, k) + at;
              if constexpr (VEC) x[u][k] = ld_cluster4(a);
              else { x[u][k].x = ld_cluster(a); x[u][k].y = ld_cluster(a + 4 * stride); x[u][k].z = ld_cluster(a + 8 * stride); x[u][k].w = ld_cluster(a + 12 * stride); }
            }
          }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
          if (!ok[u]) continue;
          v[u][0] = v[u][1] = v[u][2] = v[u][3] = 0.f;
#pragma unroll
          for (uint32_t k = 0; k < 8; ++k) { v[u][0] += x[u][k].x; v[u][1] += x[u][k].y; v[u][2] += x[u][k].z; v[u][3] += x[u][k].w; }
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (!ok[u]) continue;
        store_row4<VEC>(p, v[u], batch_off + (uint64_t)(m0 + r0 + u * step) * p.ldc, col, stride, bias, c[u], mk[u]);
#pragma unroll
        for (int j = 0; j < 4; ++j) cs[j] += v[u][j];
      }
    }
    if (p.colsum) {
#pragma unroll
      for (int j = 0; j < 4; ++j) tile[kBM * PITCH + threadIdx.x / CG * BN + local + j * stride] = cs[j];
    }
  }
  if (p.colsum) {
    __syncthreads();
    if (threadIdx.x < BN && n0 + threadIdx.x < p.n) {
      float s = 0.f;
      for (int w = 0; w < NT / CG; ++w) s += tile[kBM * PITCH + w * BN + threadIdx.x];
      atomicAdd(p.colsum + n0 + threadIdx.x, s);
    }
  }
}

template <int BN, bool A_KMAJOR, bool B_KMAJOR, int MODE, bool DIRECT = false>
__global__ void __launch_bounds__((SmemLayout<BN, MODE>::kThreads + (DIRECT ? kLoadWarps * 32 : 0)), 1)
gemm_tc_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const __grid_constant__ CUtensorMap tmC,
               const Params p) {
  static_assert(!DIRECT || MODE == kFP32X3, "direct operands: FP32X3 only");
  using MT = ModeTraits<MODE>;
  using SL = SmemLayout<BN, MODE>;
  constexpr int S = SL::kStages;
  constexpr bool X3 = (MODE == kFP32X3), SUMS = (MODE == kBF16Sums);
  // an A operand in tensor memory is K-major by construction (row m in lane m, one k element per column)
  constexpr uint32_t kIdesc = make_idesc(MT::kBf16, X3 ? false : !A_KMAJOR, !B_KMAJOR, BN);
  constexpr uint32_t kTmemCols = SL::kTmemCols;

  extern __shared__ uint8_t smem_raw[];
  // stages need 1024-byte alignment (swizzle atoms)
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint8_t* stage_base = smem;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + S * SL::kStageBytes + SL::kEpiBytes);
  uint64_t* full = bars;            // [S] TMA bytes landed
  uint64_t* ready = bars + S;       // [S] (X3) split done
  uint64_t* empty = bars + 2 * S;   // [S] MMAs that read the stage retired
  uint64_t* accum = bars + 3 * S;   // accumulator complete
  uint64_t* part_full = accum + 1;  // [2] (SUMS) a slab's products complete
  uint64_t* part_empty = accum + 3; // [2] (SUMS) ... and added up
  __shared__ uint32_t tmem_base_slot;
  __shared__ volatile int failed;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // the splits of a tile are neighbours where they form a cluster; else the tiles are, which share their slabs of A in L2
  const uint32_t tile_n = p.cluster ? blockIdx.x / p.splits : blockIdx.x % p.tiles_n;
  const uint32_t split = p.cluster ? blockIdx.x % p.splits : blockIdx.x / p.tiles_n, tile_m = blockIdx.y, batch = blockIdx.z;
  const uint32_t k_begin = split * p.k_per_split;
  uint32_t k_end = k_begin + p.k_per_split;
  if (k_end > p.k) k_end = p.k;
  const int KT = (k_end > k_begin) ? (int)((k_end - k_begin + MT::kBK - 1) / MT::kBK) : 0;

  if (threadIdx.x == 0) {
    failed = 0;
    for (int s = 0; s < S; ++s) {
      mbar_init(&full[s], DIRECT ? 1 + kLoadWarps * 32 : 1);  // the TMA thread, and every loader thread's copies
      mbar_init(&ready[s], kSplitThreads / 32);  // one arrival per split warp (of the slab's set)
      mbar_init(&empty[s], 1);
    }
    mbar_init(accum, 1);
    if constexpr (SUMS) {
      for (int i = 0; i < 2; ++i) {
        mbar_init(&part_full[i], 1);
        mbar_init(&part_empty[i], 4);
      }
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    prefetch_tmap(&tmA);
    prefetch_tmap(&tmB);
    if (p.tma_epilogue) prefetch_tmap(&tmC);
  }
  if (warp == 1) {
    tmem_alloc(&tmem_base_slot, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_d = tmem_base_slot;
  pdl_sync();  // everything above overlaps the previous kernel's tail

  if (warp == 0) {
    // ------------------------------------------------------------ producer
    if (lane == 0) {
      const int za = (int)(batch % p.nA), zb = (int)(batch % p.nB);
      for (int kt = 0; kt < KT; ++kt) {
        const int s = kt % S;
        if (kt >= S && !mbar_wait(&empty[s], ((kt / S) & 1) ^ 1, &failed)) break;
        uint8_t* st = stage_base + s * SL::kStageBytes;
        uint8_t* a_dst = st;
        uint8_t* b_dst = st + SL::kABytes;
        const bool a_tma = !DIRECT || !p.a_direct, b_tma = !DIRECT || !p.b_direct;
        mbar_expect_tx(&full[s], (a_tma ? SL::kABytes : 0) + (b_tma ? SL::kBBytes : 0));
        const int k0 = (int)k_begin + kt * MT::kBK;
        if (a_tma) {
          if (A_KMAJOR) {
            tma_load_3d(a_dst, &tmA, &full[s], k0, (int)(tile_m * kBM), za);
          } else {
#pragma unroll
            for (int j = 0; j < kBM / MT::kAtomMN; ++j)
              tma_load_3d(a_dst + j * MT::kBK * kSlabBytes, &tmA, &full[s], (int)(tile_m * kBM) + j * MT::kAtomMN, k0, za);
          }
        }
        if (b_tma) {
          if (B_KMAJOR) {
            tma_load_3d(b_dst, &tmB, &full[s], k0, (int)(tile_n * BN), zb);
          } else {
#pragma unroll
            for (int j = 0; j < BN / MT::kAtomMN; ++j)
              tma_load_3d(b_dst + j * MT::kBK * kSlabBytes, &tmB, &full[s], (int)(tile_n * BN) + j * MT::kAtomMN, k0, zb);
          }
        }
      }
    }
  } else if (DIRECT && warp >= SL::kThreads / 32) {
    // ------------------------------------------------- loaders of direct operands
    // A thread's arrival on `full` is triggered by the completion of its own copies; the split warps, which read
    // every word of B and A, order them before the tensor core's reads (fence.proxy.async before `ready`).
    if constexpr (DIRECT) {
      const float* a = p.a_src + (uint64_t)(batch % p.nA) * p.a_batch;
      const float* b = p.b_src + (uint64_t)(batch % p.nB) * p.b_batch;
      const uint32_t rows_a = p.swap ? p.n : p.m, rows_b = p.swap ? p.m : p.n;
      for (int kt = 0; kt < KT; ++kt) {
        const int s = kt % S;
        if (kt >= S) {
          const bool got = mbar_wait(&empty[s], ((kt / S) & 1) ^ 1, &failed);
          if (!__all_sync(0xffffffffu, got)) break;
        }
        uint8_t* st = stage_base + s * SL::kStageBytes;
        const uint32_t k0 = k_begin + kt * MT::kBK;
        if (p.a_direct) direct_slab<kBM, A_KMAJOR>(st, a, p.a_ld, tile_m * kBM, rows_a, k0, p.k);
        if (p.b_direct) direct_slab<BN, B_KMAJOR>(st + SL::kABytes, b, p.b_ld, tile_n * BN, rows_b, k0, p.k);
        asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(&full[s])) : "memory");
      }
      asm volatile("cp.async.wait_all;" ::: "memory");
    }
  } else if (warp == 1) {
    // ---------------------------------------------------------- MMA issuer
    // The whole warp walks the loop (waits and descriptor arithmetic stay
    // warp-uniform); one elected lane issues the MMAs and their commit.
    // The barrier of the next slab is polled once before this slab's MMAs go
    // out, so that in steady state no wait sits between two slabs.
    {
      bool have = false;
      for (int kt = 0; kt < KT; ++kt) {
        const int s = kt % S;
        if (!have) {
          const bool got = mbar_wait(X3 ? &ready[s] : &full[s], (kt / S) & 1, &failed);
          if (!__all_sync(0xffffffffu, got)) break;
        }
        bool next_seen = false;  // consumed after the MMAs of this slab are out
        if (kt + 1 < KT) {
          const int s1 = (kt + 1) % S;
          next_seen = mbar_test(X3 ? &ready[s1] : &full[s1], ((kt + 1) / S) & 1);
        }
        tc_fence_after();
        uint8_t* st = stage_base + s * SL::kStageBytes;
        const uint32_t a_hi = smem_u32(st);
        const uint32_t b_hi = a_hi + SL::kABytes, b_lo = b_hi + SL::kBBytes;
        const uint32_t a_tm = tmem_d + SL::kAccCols + (uint32_t)s * SL::kATmemCols;  // FP32X3: hi at +0, lo at +32
        // K-major: the next MMA starts 32 bytes further inside the 128-byte rows;
        // MN-major: kUmmaK k-rows (128 bytes each) further.  MN-major 32-bit
        // operands use the 32-byte-atom swizzle with 4-row groups.
        constexpr uint32_t a_step = (A_KMAJOR ? 32u : (uint32_t)(MT::kUmmaK * kSlabBytes)) >> 4;
        constexpr uint32_t b_step = (B_KMAJOR ? 32u : (uint32_t)(MT::kUmmaK * kSlabBytes)) >> 4;
        constexpr uint32_t a_lbo = A_KMAJOR ? 16u : (uint32_t)(MT::kBK * kSlabBytes);
        constexpr uint32_t b_lbo = B_KMAJOR ? 16u : (uint32_t)(MT::kBK * kSlabBytes);
        constexpr uint32_t a_lay = (!A_KMAJOR && !MT::kBf16) ? 1u : 2u, b_lay = (!B_KMAJOR && !MT::kBf16) ? 1u : 2u;
        constexpr uint32_t a_h32 = desc_hi32(a_lay == 1u ? 512u : 1024u, a_lay), b_h32 = desc_hi32(b_lay == 1u ? 512u : 1024u, b_lay);
        const uint32_t da0 = desc_lo32(a_hi, a_lbo);
        const uint32_t db0 = desc_lo32(b_hi, b_lbo), dbl0 = desc_lo32(b_lo, b_lbo);
        // Every instruction truncates its accumulator once.  The two small products of three passes add up in an accumulator of
        // their own, where a truncation is 2^-11 of one of the sum, and the large one is cut a third as often: 494x1150x1037 in four
        // K ranges 4.0e-6 off in the 2-norm, 1.5e-6 like this, 1681x1161x6503 in one 4.6e-5 and 1.6e-5, 51 random shapes in
        // the same time within 2 %.
        if (elect_one()) {
#pragma unroll
        for (int kk = 0; kk < MT::kBK / MT::kUmmaK; ++kk) {
          const uint64_t db = desc_pack(db0 + kk * b_step, b_h32);
          const uint32_t acc = (kt > 0 || kk > 0) ? 1u : 0u;
          if constexpr (X3) {
            const uint64_t dbl = desc_pack(dbl0 + kk * b_step, b_h32);
            const uint32_t ta_hi = a_tm + kk * MT::kUmmaK, ta_lo = ta_hi + 32, small = tmem_d + SL::kAccOne;
            umma_tmem_a(small, ta_lo, db, kIdesc, acc);    // Alo * Bhi
            umma_tmem_a(small, ta_hi, dbl, kIdesc, 1u);    // Ahi * Blo
            umma_tmem_a(tmem_d, ta_hi, db, kIdesc, acc);   // Ahi * Bhi
          } else {
            const uint64_t da = desc_pack(da0 + kk * a_step, a_h32);
            if constexpr (SUMS) {
              const int part = (kt * (MT::kBK / MT::kUmmaK) + kk) / SL::kInPart, at = kk % SL::kInPart;
              if (at == 0 && part >= 2 && !mbar_wait(&part_empty[part & 1], ((part >> 1) & 1) ^ 1, &failed)) break;
              umma<MT::kBf16>(tmem_d + (part & 1) * SL::kAccOne, da, db, kIdesc, at > 0 ? 1u : 0u);
              if (at == SL::kInPart - 1) umma_commit(&part_full[part & 1]);
            } else umma<MT::kBf16>(tmem_d, da, db, kIdesc, acc);
          }
        }
        umma_commit(&empty[s]);  // stage reusable once these MMAs have read it
        }
        have = __all_sync(0xffffffffu, next_seen);
      }
      if (elect_one()) umma_commit(accum);
    }
  } else if constexpr (X3) {
    // ------------------------------------------- hi/lo split (warps 2..7)
    const int t = threadIdx.x - 64;
    const bool a_warp = warp >= 4;  // the two times four warps that cover the TMEM lane quadrants (warp % 4)
    if (a_warp) {
      // Four warps (TMEM lane quadrant = warp % 4), thread = row of the A slab.  The row's eight
      // 16-byte chunks sit at chunk position c ^ (row % 8) (128-byte swizzle); hi = the fetched
      // word itself, lo = x - tf32(x); both go to tensor memory.  The row of the NEXT slab is
      // fetched while the stores of this one drain, so a warp's chain per slab is
      // split -> store -> (load next) -> wait -> arrive.
      const int row = (warp & 3) * 32 + lane;
      const uint32_t ta0 = tmem_d + SL::kAccCols + ((uint32_t)((warp & 3) * 32) << 16);
      float4 v[8];
      bool have = false;
      auto load_row = [&](int stage) { load_a_row<A_KMAJOR>(stage_base + stage * SL::kStageBytes, row, v); };
      for (int kt = warp >= 8 ? 1 : 0; kt < KT; kt += 2) {
        const int s = kt % S;
        if (!have) {
          const bool got = mbar_wait(&full[s], (kt / S) & 1, &failed);
          if (!__all_sync(0xffffffffu, got)) break;
          load_row(s);
        }
        uint32_t hi[32], lo[32];
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          const float x[4] = {v[c].x, v[c].y, v[c].z, v[c].w};
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const uint32_t h = __float_as_uint(x[e]) & 0xFFFFE000u;
            hi[4 * c + e] = __float_as_uint(x[e]);
            lo[4 * c + e] = __float_as_uint(x[e] - __uint_as_float(h));
          }
        }
        const uint32_t ta = ta0 + (uint32_t)s * SL::kATmemCols;
        tmem_st32(ta, hi);
        tmem_st32(ta + 32, lo);
        if constexpr (SL::kBWordsA > 0) {
          // this warp's share of the B split (the words after those of the two B warps)
          float4* bh = reinterpret_cast<float4*>(stage_base + s * SL::kStageBytes + SL::kABytes);
          float4* bl = bh + SL::kBBytes / 16;
#pragma unroll
          for (int j = 0; j < SL::kBWordsA; ++j) {
            const int i = 64 * SL::kBWordsB + (threadIdx.x & 127) + 128 * j;
            const float4 b = bh[i];
            float4 l;
            l.x = b.x - __uint_as_float(__float_as_uint(b.x) & 0xFFFFE000u);
            l.y = b.y - __uint_as_float(__float_as_uint(b.y) & 0xFFFFE000u);
            l.z = b.z - __uint_as_float(__float_as_uint(b.z) & 0xFFFFE000u);
            l.w = b.w - __uint_as_float(__float_as_uint(b.w) & 0xFFFFE000u);
            bl[i] = l;
          }
        }
        have = false;
        if (kt + 2 < KT) {
          const int s2 = (kt + 2) % S;
          have = __all_sync(0xffffffffu, mbar_test(&full[s2], ((kt + 2) / S) & 1));
          if (have) load_row(s2);
        }
        if constexpr (SL::kBWordsA > 0) fence_async_smem();
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&ready[s]);
      }
    } else {
      // The two other warps split B: lo = x - tf32(x) into the second B buffer of the stage.
      // Like the A warps they fetch the next slab's part before they hand this one over.
      constexpr int NB = SL::kBWordsB;  // 16-byte words per thread and slab
      float4 v[NB];
      bool have = false;
      auto b_hi_of = [&](int stage) { return reinterpret_cast<float4*>(stage_base + stage * SL::kStageBytes + SL::kABytes); };
      auto load_b = [&](int stage) {
        const float4* src = b_hi_of(stage);
#pragma unroll
        for (int j = 0; j < NB; ++j) v[j] = src[t + 64 * j];
      };
      for (int kt = 0; kt < KT; ++kt) {
        const int s = kt % S;
        if (!have) {
          const bool got = mbar_wait(&full[s], (kt / S) & 1, &failed);
          if (!__all_sync(0xffffffffu, got)) break;
          load_b(s);
        }
        float4* dst = b_hi_of(s) + SL::kBBytes / 16;
#pragma unroll
        for (int j = 0; j < NB; ++j) {
          float4 l;
          l.x = v[j].x - __uint_as_float(__float_as_uint(v[j].x) & 0xFFFFE000u);
          l.y = v[j].y - __uint_as_float(__float_as_uint(v[j].y) & 0xFFFFE000u);
          l.z = v[j].z - __uint_as_float(__float_as_uint(v[j].z) & 0xFFFFE000u);
          l.w = v[j].w - __uint_as_float(__float_as_uint(v[j].w) & 0xFFFFE000u);
          dst[t + 64 * j] = l;
        }
        have = false;
        if (kt + 1 < KT) {
          const int s1 = (kt + 1) % S;
          have = __all_sync(0xffffffffu, mbar_test(&full[s1], ((kt + 1) / S) & 1));
          if (have) load_b(s1);
        }
        fence_async_smem();  // generic-proxy writes -> visible to the tensor core's async proxy
        __syncwarp();
        if (lane == 0) mbar_arrive(&ready[s]);
      }
    }
  }

  // ---------------------------------------------------------------- epilogue
  // Each of these threads owns one accumulator row and takes 32 consecutive columns of it per tcgen05.ld: into swizzled
  // boxes for the TMA unit, or into the staged tile that all warps then finish.
  if (warp >= 4 && warp < 8) {
    const int q = warp - 4;  // TMEM lane quadrant
    bool have_acc = KT > 0;
    if constexpr (SUMS) {
      // The parts of the sum are added up here, rounding to nearest, and take the accumulator's place.  64-wide tiles carry what
      // each addition rounds off to the next one (Kahan's summation).
      constexpr bool CARRY = BN == 64;
      const uint32_t at = tmem_d + ((uint32_t)(q * 32) << 16);
      float sum[BN], off[CARRY ? BN : 1];
#pragma unroll
      for (int j = 0; j < BN; ++j) {
        sum[j] = 0.f;
        if constexpr (CARRY) off[j] = 0.f;
      }
      const int parts = KT * (MT::kBK / MT::kUmmaK) / SL::kInPart;
      for (int part = 0; part < parts; ++part) {
        const bool got = mbar_wait(&part_full[part & 1], (part >> 1) & 1, &failed);
        if (!__all_sync(0xffffffffu, got)) { have_acc = false; break; }
        tc_fence_after();
#pragma unroll
        for (int c = 0; c < BN; c += 64) {
          uint32_t r[32], t[32];
          tmem_ld32(at + (part & 1) * SL::kAccOne + c, r);
          tmem_ld32(at + (part & 1) * SL::kAccOne + c + 32, t);
          tmem_ld_wait();
          if (c + 64 == BN) {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&part_empty[part & 1]);
          }
#pragma unroll
          for (int j = 0; j < 64; ++j) {
            const float x = __uint_as_float(j < 32 ? r[j % 32] : t[j % 32]);
            if constexpr (CARRY) {
              const float y = x - off[j], z = sum[j] + y, e = (z - sum[j]) - y;
              off[j] = fabsf(e) < INFINITY ? e : 0.f;  // (behind an infinity, or a sum that became one, there is nothing to carry)
              sum[j] = z;
            } else {
              sum[c + j] += x;
            }
          }
        }
      }
      if (have_acc) {
#pragma unroll
        for (int c = 0; c < BN; c += 32) {
          uint32_t r[32];
#pragma unroll
          for (int j = 0; j < 32; ++j) r[j] = __float_as_uint(sum[c + j]);
          tmem_st32(at + c, r);
        }
        tmem_st_wait();
      }
    } else {
      have_acc = have_acc && mbar_wait(accum, 0, &failed);
    }
    tc_fence_after();
    if (p.tma_epilogue && (KT == 0 || have_acc)) {
      // The stage ring is idle by now (every fetched slab was consumed by MMAs that have completed):
      // its first bytes stage the output, 4 KB per warp and chunk, 1024-byte aligned for the swizzle.
      uint8_t* stg = stage_base + q * (BN / 32) * 4096;
      const bool has_bias = p.epilogue == ZG_EPI_BIAS || p.epilogue == ZG_EPI_BIAS_RELU;
      int chunks = 0;
#pragma unroll 1
      for (int c = 0; c < BN / 32; ++c) {
        const uint32_t col0 = tile_n * BN + c * 32;
        if (col0 >= p.n) break;  // uniform across the warp
        uint32_t r[32];
        if (KT > 0) {
          load_accumulator<X3>(tmem_d + ((uint32_t)(q * 32) << 16) + (uint32_t)(c * 32), SL::kAccOne, r);
        } else {
#pragma unroll
          for (int j = 0; j < 32; ++j) r[j] = 0u;
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
        }
        uint8_t* rowp = stg + c * 4096 + lane * 128;
#pragma unroll
        for (int j = 0; j < 8; ++j)
          *reinterpret_cast<float4*>(rowp + ((j ^ (lane & 7)) << 4)) = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
        ++chunks;
      }
      fence_async_smem();  // generic-proxy writes -> visible to the TMA unit
      __syncwarp();
      if (lane == 0 && tile_m * kBM + q * 32 < p.m) {
        for (int c = 0; c < chunks; ++c) {
          const int x = (int)(tile_n * BN) + c * 32, y = (int)(tile_m * kBM) + q * 32;
          if (p.tma_epilogue == 2) tma_reduce_add_box(&tmC, stg + c * 4096, x, y, (int)batch);
          else tma_store_box(&tmC, stg + c * 4096, x, y, (int)batch);
        }
        bulk_commit_group();
        bulk_wait_group_read();
      }
      __syncwarp();
    } else if (KT == 0 || have_acc) {
      // Row q * 32 + lane of the tile into the idle ring: 16-byte words whose 4-bank row offset keeps the eight rows
      // of a quarter-warp apart.
      float* rowp = reinterpret_cast<float*>(stage_base) + (q * 32 + lane) * SL::kOutPitch;
#pragma unroll 1
      for (int c = 0; c < BN / 32; ++c) {
        uint32_t r[32];
        if (KT > 0) {
          load_accumulator<X3>(tmem_d + ((uint32_t)(q * 32) << 16) + (uint32_t)(c * 32), SL::kAccOne, r);  // warp-collective
        } else {
#pragma unroll
          for (int j = 0; j < 32; ++j) r[j] = 0u;
        }
#pragma unroll
        for (int j = 0; j < 32; j += 4) *reinterpret_cast<uint4*>(rowp + c * 32 + j) = make_uint4(r[j], r[j + 1], r[j + 2], r[j + 3]);
      }
    }
  }
  __syncwarp();
  if (!p.tma_epilogue) {
    float* tile = reinterpret_cast<float*>(stage_base);
    if (p.cluster) cluster_sync(); else __syncthreads();
    constexpr int NT = SL::kThreads + (DIRECT ? kLoadWarps * 32 : 0);
    const uint64_t batch_off = (uint64_t)batch * p.c_batch_stride;
    if (p.swap) staged_out_swapped<BN, NT>(p, tile, split, tile_m * kBM, tile_n * BN, batch_off);
    else if (p.vec_ok && (p.n & 3u) == 0) {
      if (p.cluster) staged_out<BN, NT, true, 1>(p, tile, split, tile_m * kBM, tile_n * BN, batch_off);
      else staged_out<BN, NT, true, 2>(p, tile, split, tile_m * kBM, tile_n * BN, batch_off);
    } else {
      if (p.cluster) staged_out<BN, NT, false, 1>(p, tile, split, tile_m * kBM, tile_n * BN, batch_off);
      else staged_out<BN, NT, false, 2>(p, tile, split, tile_m * kBM, tile_n * BN, batch_off);
    }
    if (p.cluster) cluster_sync();  // nobody leaves while its partial tile may still be read
  }

  // ---------------------------------------------------------------- teardown
  tc_fence_before();
  __syncthreads();
  if (failed) outstay_own_work();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_d, kTmemCols);
  }
  if (threadIdx.x == 0 && failed && p.error_flag) *p.error_flag = 1;
}

}  // namespace tc
}  // namespace zg

// FFMA / DFMA matrix product for problems the tensor-core kernels do not take: small ones (the layers of
// an MLP at batch 1 .. a few hundred), fp64, and operands whose rows no TMA box can address.
//
//   C[b] = epilogue(alpha * op(A[b % nA]) * op(B[b % nB]) + beta * C[b])
//
// What bounds the small problems is latency, not arithmetic: a 64x128x784 product is 6.4 M multiply-adds
// (0.4 us of the chip's FFMA rate) behind one memory round trip.  So the k dimension is cut three times:
//   * over the CTAs of a thread-block cluster (up to 8), whose partial tiles are summed through
//     distributed shared memory in rank order -- one launch, no atomics, no pre-scaled C, and every
//     epilogue (bias, ReLU, mask, column sums) still applies to the finished sums;
//   * over KG groups of threads inside the CTA, folded through shared memory;
//   * over a ring of kStages asynchronous copies, so that a CTA's whole k range (64-deep slabs) is
//     in flight after its first few instructions.
// Element-wise cp.async (4 or 8 bytes) needs no alignment beyond the element's own and transposes on the
// way into shared memory: both operands are kept [k][row], so a thread's operands are 16-byte reads.
// Measured (operands in L2, one launch of a replayed chain): 64x128x784 + bias + ReLU 4.1 us (13.8 as 5 K splits of
// one 128-row tensor-core tile, 49.7 for one row on the 64x64 tile kernel this one replaced), 128x784x64 4.8 (7.9),
// 64x10x64 3.1 (6.3), 1000x501x1000 unaligned 49 (66).  fp64 with more than half a
// 64x64 tile per SM runs in gemm_f64.cuh, but for the shortest sums.
#pragma once

#include <cooperative_groups.h>

#include "common.cuh"

namespace zg {
namespace block {

constexpr int kThreads = 256;

template <typename T> struct Acc { using type = float; };
template <> struct Acc<double> { using type = double; };

template <typename T> __device__ __forceinline__ typename Acc<T>::type to_acc(T v) { return (typename Acc<T>::type)v; }
template <> __device__ __forceinline__ float to_acc<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }
template <typename TC, typename A> __device__ __forceinline__ TC from_acc(A v) { return (TC)v; }
template <> __device__ __forceinline__ __nv_bfloat16 from_acc<__nv_bfloat16, float>(float v) { return __float2bfloat16_rn(v); }

struct Params {
  uint64_t nA, nB, m, n, k, lda, ldb, ldc, a_stride, b_stride, c_stride;
  double alpha, beta;
  const float* bias;
  const void* mask;
  float* colsum;
  uint64_t k_per_split;  // k range of one CTA of a cluster
  uint32_t splits;       // cluster size
  uint32_t tiles_m, tiles_n;
  int ta, tb;
  int epilogue;
};

// One weight gradient of a grouped launch: C[m, n] = A^T B over the rows of a batch (p.ta, p.beta = 0), with A's column sums.
// Each of C, colsum, W and b may be missing.  W += nlr * C, b += nlr * column sums (the SGD step, once the sums are final).
constexpr int kGroupMax = 6;
struct GroupItem {
  const float *A, *B;
  float *C, *W, *colsum, *b;
  uint32_t m, n, lda, ldb, tiles_n;
  uint32_t first;  // its first output tile in the launch
};
struct Group {
  GroupItem item[kGroupMax];
  uint32_t items, k, k_per_split, splits;
  float nlr;
};

// Tile TM x TN of C per cluster.  MI x MI outputs per thread: TM * TN / MI^2 threads make one k group.  MI == 0: fp64 on
// the tensor cores, 32 x 32 outputs per warp.
template <typename TI, int TM, int TN, int MI>
struct Layout {
  using AT = typename Acc<TI>::type;
  static constexpr int kGroupThreads = MI ? TM * TN / (MI * MI + (MI == 0)) : TM * TN / 32;
  static constexpr int KG = kThreads / kGroupThreads;
  static constexpr int TK = sizeof(AT) == 8 ? 32 : 64;  // k depth of a stage
  static constexpr int kPerGroup = TK / KG;
  // 16-byte aligned rows; 8 k x 4 rows of a copy hit 32 banks, and so do the 4 k x 8 rows of an fp64 fragment
  static constexpr int kPadA = TM + 4, kPadB = TN + 4;
  static constexpr int kStageElems = TK * (kPadA + kPadB);
  static constexpr int kStages = sizeof(TI) < 4 ? 2 : 3;
  static constexpr size_t kRedBytes = (size_t)KG * TM * TN * sizeof(AT);
  static constexpr size_t kRingBytes = (size_t)kStages * kStageElems * sizeof(AT);
  static constexpr size_t kSmem = kRingBytes > kRedBytes ? kRingBytes : kRedBytes;
};

template <int BYTES>
__device__ __forceinline__ void copy_async(void* smem, const void* gmem, bool ok) {
  const uint32_t dst = (uint32_t)__cvta_generic_to_shared(smem);
  const int n = ok ? BYTES : 0;  // 0 source bytes: the destination is filled with zeros
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(dst), "l"(gmem), "n"(BYTES), "r"(n) : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// One operand's side of the copies.  Thread t moves elements (row0 + i * drow, k0 + i * dk) of every ROWS x TK slab: a
// source that is contiguous in k is read 8 consecutive k (one 32-byte sector of fp32) of 4 rows per warp, one that is
// contiguous in its rows 32 rows of one k.  Either way the source and the destination of consecutive i are a
// constant apart, so a copy costs an add and a compare.
template <typename T, int ROWS, int TK, int PAD>
struct Copier {
  static constexpr int N = ROWS * TK / kThreads;
  const T* src;    // element (row0, k0) of the next slab
  int64_t step;    // source distance between consecutive i
  int64_t advance; // source distance between consecutive slabs
  int row0, kk0, drow, dk;
  int rows, dst0, ddst;
  __device__ __forceinline__ void init(const T* base, bool k_contig, uint64_t first_row, uint64_t row_count, uint64_t first_k, uint64_t ld) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    constexpr int W = kThreads / 32;
    if (k_contig) {
      constexpr int KB = TK / 8;  // 8-wide k blocks; W is a multiple of KB
      kk0 = (w % KB) * 8 + (lane & 7);
      row0 = (w / KB) * 4 + (lane >> 3);
      drow = W / KB * 4;
      dk = 0;
      step = (int64_t)drow * (int64_t)ld;
      advance = TK;
      src = base + (int64_t)(first_row + row0) * (int64_t)ld + (int64_t)(first_k + kk0);
    } else {
      constexpr int RB = ROWS / 32;
      row0 = (w % RB) * 32 + lane;
      kk0 = w / RB;
      drow = 0;
      dk = W / RB;
      step = (int64_t)dk * (int64_t)ld;
      advance = (int64_t)TK * (int64_t)ld;
      src = base + (int64_t)(first_k + kk0) * (int64_t)ld + (int64_t)(first_row + row0);
    }
    const uint64_t r = row_count > first_row ? row_count - first_row : 0;
    rows = r < (uint64_t)ROWS ? (int)r : ROWS;
    dst0 = kk0 * PAD + row0;
    ddst = dk * PAD + drow;
  }
  __device__ __forceinline__ bool ok(int i, int k_left) const { return row0 + i * drow < rows && kk0 + i * dk < k_left; }
};

template <typename T>
__device__ __forceinline__ void load4(const T* p, T (&v)[4]) {
  if constexpr (sizeof(T) == 4) {
    const float4 x = *reinterpret_cast<const float4*>(p);
    v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
  } else {
    const double2 x = *reinterpret_cast<const double2*>(p), y = *reinterpret_cast<const double2*>(p + 2);
    v[0] = x.x; v[1] = x.y; v[2] = y.x; v[3] = y.y;
  }
}

// D (8 x 8) += A (8 x 4) * B (4 x 8) in fp64: lane l holds A[l / 4][l % 4], B[l % 4][l / 4] and D[l / 4][2 (l % 4)], [.. + 1].
// Against DFMA it halves the shared-memory reads per multiply-add.
__device__ __forceinline__ void mma_f64(double (&d)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};" : "+d"(d[0]), "+d"(d[1]) : "d"(a), "d"(b));
}

// GROUP: `item` of a grouped launch, whose A has its column sums formed from the slabs as they pass.
template <typename TI, typename TC, int TM, int TN, int MI, bool GROUP = false>
__device__ __forceinline__ void block_tile(const TI* __restrict__ A, const TI* __restrict__ B, TC* C, const Params& p, const uint32_t split, uint32_t tile,
                                           const GroupItem& item, const float nlr) {
  static_assert(!GROUP || (TM == 32 && TN == 32), "the column sums of a grouped launch");
  using L = Layout<TI, TM, TN, MI>;
  using AT = typename L::AT;
  constexpr int KG = L::KG, TK = L::TK, S = L::kStages;
  constexpr bool kAsync = sizeof(TI) >= 4;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  AT* ring = reinterpret_cast<AT*>(smem_raw);
  __shared__ float col_part[kThreads / TN][TN];

  __shared__ float row_part[GROUP ? 8 : 1][32], row_total[32];
  const uint32_t tn = tile % p.tiles_n;
  tile /= p.tiles_n;
  const uint32_t tm = tile % p.tiles_m;
  const uint64_t batch = tile / p.tiles_m;
  const uint64_t m0 = (uint64_t)tm * TM, n0 = (uint64_t)tn * TN;
  const uint64_t kb = split * p.k_per_split;
  const uint64_t ke = kb + p.k_per_split < p.k ? kb + p.k_per_split : p.k;
  const int depth = ke > kb ? (int)(ke - kb) : 0;
  const int chunks = (depth + TK - 1) / TK;
  Copier<TI, TM, TK, L::kPadA> ca;
  Copier<TI, TN, TK, L::kPadB> cb;
  ca.init(A + (batch % p.nA) * p.a_stride, !p.ta, m0, p.m, kb, p.lda);
  cb.init(B + (batch % p.nB) * p.b_stride, p.tb != 0, n0, p.n, kb, p.ldb);

  // cp.async of the next slab into stage c % S; always one commit group, so that the waits below count slabs
  auto issue = [&](int c) {
    if (c < chunks) {
      AT* as = ring + (c % S) * L::kStageElems;
      AT* bs = as + TK * L::kPadA;
      const int left = depth - c * TK;
      if constexpr (kAsync) {
#pragma unroll
        for (int i = 0; i < ca.N; ++i) {
          const bool ok = ca.ok(i, left);
          copy_async<(int)sizeof(TI)>(as + ca.dst0 + i * ca.ddst, ok ? ca.src + i * ca.step : A, ok);
        }
#pragma unroll
        for (int i = 0; i < cb.N; ++i) {
          const bool ok = cb.ok(i, left);
          copy_async<(int)sizeof(TI)>(bs + cb.dst0 + i * cb.ddst, ok ? cb.src + i * cb.step : B, ok);
        }
        ca.src += ca.advance;
        cb.src += cb.advance;
      }
    }
    if constexpr (kAsync) copy_commit();
  };
  // 16-bit inputs: widened in registers on their way to shared memory
  AT ra[kAsync ? 1 : ca.N], rb[kAsync ? 1 : cb.N];
  auto fetch = [&](int c) {
    if constexpr (!kAsync) {
      const int left = depth - c * TK;
#pragma unroll
      for (int i = 0; i < ca.N; ++i) ra[i] = ca.ok(i, left) ? to_acc<TI>(ca.src[i * ca.step]) : AT(0);
#pragma unroll
      for (int i = 0; i < cb.N; ++i) rb[i] = cb.ok(i, left) ? to_acc<TI>(cb.src[i * cb.step]) : AT(0);
      ca.src += ca.advance;
      cb.src += cb.advance;
    }
  };
  auto park = [&](int c) {
    if constexpr (!kAsync) {
      AT* as = ring + (c % S) * L::kStageElems;
      AT* bs = as + TK * L::kPadA;
#pragma unroll
      for (int i = 0; i < ca.N; ++i) as[ca.dst0 + i * ca.ddst] = ra[i];
#pragma unroll
      for (int i = 0; i < cb.N; ++i) bs[cb.dst0 + i * cb.ddst] = rb[i];
    }
  };

  const int group = threadIdx.x / L::kGroupThreads, gt = threadIdx.x % L::kGroupThreads;
  // rows ty * 4 + (i / 4) * TM / 2 + i % 4, columns likewise: 16-byte reads, consecutive threads on consecutive words
  constexpr int MIN = MI ? MI : 4;  // (fp64: 4 x 4 blocks of 8 x 8 per warp)
  const int tx = MI ? gt % (TN / MIN) : gt / 32 % (TN / 32), ty = MI ? gt / (TN / MIN) : gt / 32 / (TN / 32);
  const int lane = threadIdx.x & 31;
  AT acc[MI ? MIN : 1][MI ? MIN : 1];
  double dacc[MI ? 1 : 4][MI ? 1 : 4][2];
  if constexpr (MI == 0) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) dacc[i][j][0] = dacc[i][j][1] = 0.0;
  } else {
#pragma unroll
    for (int i = 0; i < MI; ++i)
#pragma unroll
      for (int j = 0; j < MI; ++j) acc[i][j] = AT(0);
  }

  // GROUP: a slab's sums of 16 products are added up in a second set of registers.  All layers share the launch's number of K
  // ranges, fewer than a small one has by itself, and one chain over the longer ranges was up to 1.3 times as far off (100
  // random networks: 1.08 times the error of the products one by one on average, 0.94 like this, in the same time).
  AT total[GROUP ? MI : 1][GROUP ? MI : 1];
  if constexpr (GROUP) {
#pragma unroll
    for (int i = 0; i < MI; ++i)
#pragma unroll
      for (int j = 0; j < MI; ++j) total[i][j] = AT(0);
  }
  const bool sums = GROUP && tn == 0 && (item.colsum || item.b);
  float rsum = 0.f;
  pdl_sync();
  if constexpr (kAsync) {
#pragma unroll
    for (int c = 0; c < S - 1; ++c) issue(c);
  } else if (chunks > 0) {
    fetch(0);
    park(0);
    if (chunks > 1) fetch(1);
  }
  for (int c = 0; c < chunks; ++c) {
    if constexpr (kAsync) copy_wait<S - 2>();
    __syncthreads();  // slab c has landed; everyone is done with slab c - 1, whose stage the next copy reuses
    if constexpr (kAsync) issue(c + S - 1);
    const AT* as = ring + (c % S) * L::kStageElems + group * L::kPerGroup * L::kPadA + ty * (MI ? 4 : 32);
    const AT* bs = ring + (c % S) * L::kStageElems + TK * L::kPadA + group * L::kPerGroup * L::kPadB + tx * (MI ? 4 : 32);
    const int left = depth - c * TK - group * L::kPerGroup;
    if constexpr (GROUP) {  // (rows past k are zeros)
      if (sums) {
        const AT* a0 = ring + (c % S) * L::kStageElems + (threadIdx.x & 31);
#pragma unroll
        for (int kk = 0; kk < TK; kk += 8) rsum += a0[(kk + (threadIdx.x >> 5)) * L::kPadA];
      }
    }
    if constexpr (MI == 0) {
      if (left > 0) {  // the slab is padded with zeros
#pragma unroll
        for (int kk = 0; kk < L::kPerGroup; kk += 4) {
          double av[4], bv[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            av[i] = as[(kk + lane % 4) * L::kPadA + 8 * i + lane / 4];
            bv[i] = bs[(kk + lane % 4) * L::kPadB + 8 * i + lane / 4];
          }
#pragma unroll
          for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) mma_f64(dacc[i][j], av[i], bv[j]);
        }
      }
    } else {
      auto mac = [&](int kk) {
        AT av[MIN], bv[MIN];
#pragma unroll
        for (int h = 0; h < MI / 4; ++h) {
          load4(as + kk * L::kPadA + h * (TM / 2), *reinterpret_cast<AT(*)[4]>(av + 4 * h));
          load4(bs + kk * L::kPadB + h * (TN / 2), *reinterpret_cast<AT(*)[4]>(bv + 4 * h));
        }
#pragma unroll
        for (int i = 0; i < MI; ++i)
#pragma unroll
          for (int j = 0; j < MI; ++j) acc[i][j] += av[i] * bv[j];
      };
      if (left >= L::kPerGroup) {
#pragma unroll
        for (int kk = 0; kk < L::kPerGroup; ++kk) mac(kk);
      } else {
        for (int kk = 0; kk < left; ++kk) mac(kk);
      }
      if constexpr (GROUP) {
#pragma unroll
        for (int i = 0; i < MI; ++i)
#pragma unroll
          for (int j = 0; j < MI; ++j) {
            total[i][j] += acc[i][j];
            acc[i][j] = AT(0);
          }
      }
    }
    if constexpr (!kAsync) {
      if (c + 1 < chunks) park(c + 1);  // the other stage: its readers passed the barrier above
      if (c + 2 < chunks) fetch(c + 2);
    }
  }

  // ---- fold the k groups, then the cluster, then the epilogue; lanes run along n, so every access to C is coalesced
  constexpr int kOut = TM * TN / kThreads;  // outputs per thread
  if constexpr (kAsync) copy_wait<0>();
  __syncthreads();
  AT* red = ring;
  if constexpr (MI == 0) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j)
        *reinterpret_cast<double2*>(&red[(group * TM + ty * 32 + 8 * i + lane / 4) * TN + tx * 32 + 8 * j + lane % 4 * 2]) = make_double2(dacc[i][j][0], dacc[i][j][1]);
  } else {
#pragma unroll
    for (int i = 0; i < MI; ++i)
#pragma unroll
      for (int j = 0; j < MI; ++j)
        red[(group * TM + ty * 4 + (i / 4) * (TM / 2) + i % 4) * TN + tx * 4 + (j / 4) * (TN / 2) + j % 4] = GROUP ? total[GROUP ? i : 0][GROUP ? j : 0] : acc[i][j];
  }
  if constexpr (GROUP) row_part[threadIdx.x >> 5][threadIdx.x & 31] = rsum;
  __syncthreads();
  if constexpr (GROUP) {
    if (sums && threadIdx.x < 32) {
      float s = 0.f;
#pragma unroll
      for (int w = 0; w < 8; ++w) s += row_part[w][threadIdx.x];
      row_total[threadIdx.x] = s;
    }
  }
  AT sum[kOut];
#pragma unroll
  for (int o = 0; o < kOut; ++o) {
    sum[o] = red[threadIdx.x + o * kThreads];
#pragma unroll
    for (int g = 1; g < KG; ++g) sum[o] += red[g * TM * TN + threadIdx.x + o * kThreads];
  }
  const AT alpha = (AT)p.alpha, beta = (AT)p.beta;
  TC* c = C + batch * p.c_stride;
  float csum = 0.f;
  auto finish = [&](int e, AT v) {
    const uint64_t gm = m0 + e / TN, gn = n0 + e % TN;
    if (gm >= p.m || gn >= p.n) return;
    const uint64_t o = gm * p.ldc + gn;
    if constexpr (GROUP) {
      if (C) C[o] = v;
      if (item.W) item.W[o] = fmaf(nlr, v, item.W[o]);
      return;
    }
    v *= alpha;
    if (beta != AT(0)) v += beta * to_acc<TC>(c[o]);
    if (p.epilogue == ZG_EPI_BIAS) v += (AT)p.bias[gn];
    else if (p.epilogue == ZG_EPI_BIAS_RELU) { v += (AT)p.bias[gn]; v = v > AT(0) ? v : AT(0); }
    else if (p.epilogue == ZG_EPI_RELU_MASK) {
      const TC* mk = static_cast<const TC*>(p.mask) + batch * p.c_stride;
      if (to_acc<TC>(mk[o]) <= AT(0)) v = AT(0);
    }
    c[o] = from_acc<TC, AT>(v);
    csum += (float)v;
  };
  auto put_sum = [&](float v) {
    const uint64_t gm = m0 + threadIdx.x;
    if (gm >= p.m) return;
    if (item.colsum) item.colsum[gm] = v;
    if (item.b) item.b[gm] = fmaf(nlr, v, item.b[gm]);
  };
  if (p.splits == 1) {
#pragma unroll
    for (int o = 0; o < kOut; ++o) finish(threadIdx.x + o * kThreads, sum[o]);
    if (sums && threadIdx.x < 32) put_sum(row_total[threadIdx.x]);
  } else {
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    // each element's own thread wrote and read it above: no barrier needed before it is overwritten
#pragma unroll
    for (int o = 0; o < kOut; ++o) red[threadIdx.x + o * kThreads] = sum[o];
    cluster.sync();
    const int share = TM * TN / (int)p.splits;  // this CTA finishes one share of the tile (whole rows: splits <= 8)
    for (int e = threadIdx.x; e < share; e += kThreads) {
      const int at = (int)split * share + e;
      // all ranks' values are requested before the first is added: one round trip over the cluster network, not eight
      AT part[8], v = AT(0);
#pragma unroll
      for (uint32_t r = 0; r < 8; ++r) part[r] = r < p.splits ? cluster.map_shared_rank(red, r)[at] : AT(0);
#pragma unroll
      for (uint32_t r = 0; r < 8; ++r) v += part[r];
      finish(at, v);
    }
    if constexpr (GROUP) {
      if (sums && split == 0 && threadIdx.x < 32) {
        float v = 0.f;
        for (uint32_t r = 0; r < p.splits; ++r) v += cluster.map_shared_rank(row_total, r)[threadIdx.x];
        put_sum(v);
      }
    }
    cluster.sync();  // nobody leaves while its partial tile may still be read
  }
  if (!GROUP && p.colsum) {
    // a thread's outputs all lie in column threadIdx.x % TN: kThreads and the shares are multiples of TN
    col_part[threadIdx.x / TN][threadIdx.x % TN] = csum;
    __syncthreads();
    if (threadIdx.x < TN && n0 + threadIdx.x < p.n) {
      float s = 0.f;
#pragma unroll
      for (int w = 0; w < kThreads / TN; ++w) s += col_part[w][threadIdx.x];
      atomicAdd(p.colsum + n0 + threadIdx.x, s);
    }
  }
}

template <typename TI, typename TC, int TM, int TN, int MI>
__global__ void __launch_bounds__(kThreads, MI == 0 ? 2 : 1) gemm_block_kernel(const TI* __restrict__ A, const TI* __restrict__ B, TC* C, const Params p) {
  block_tile<TI, TC, TM, TN, MI>(A, B, C, p, blockIdx.x % p.splits, blockIdx.x / p.splits, GroupItem{}, 0.f);
}

// The weight gradients of a network on few rows, their column sums (the biases' gradients) and the SGD step in one launch:
// a tile of any of the products per cluster.  One by one they are chains of two or three launches of 2 to 4 us on streams
// forked off and joined again, behind a fill of the buffer they accumulate into: 784-128-64-10 on 64 rows
// 20.5 -> 18.4 us a step as a kept graph, 132 -> 78 us where its launches are issued one by one.
__global__ void __launch_bounds__(kThreads, 1) weight_grads_kernel(const __grid_constant__ Group g) {
  uint32_t tile = blockIdx.x / g.splits;
  int i = 0;
#pragma unroll
  for (int j = 1; j < kGroupMax; ++j)
    if (j < (int)g.items && tile >= g.item[j].first) i = j;
  const GroupItem item = g.item[i];
  Params p = {};
  p.nA = p.nB = 1;
  p.m = item.m; p.n = item.n; p.k = g.k; p.lda = item.lda; p.ldb = item.ldb; p.ldc = item.n;
  p.k_per_split = g.k_per_split; p.splits = g.splits;
  p.tiles_n = item.tiles_n; p.tiles_m = (item.m + 31) / 32;
  p.ta = 1;
  block_tile<float, float, 32, 32, 4, true>(item.A, item.B, item.C, p, blockIdx.x % g.splits, tile - item.first, item, g.nlr);
}

}  // namespace block
}  // namespace zg

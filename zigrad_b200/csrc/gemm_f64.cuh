// fp64 matrix product on the double-precision tensor instruction (mma.sync m16n8k8), persistent and warp-specialised.
//
//   C[b] = epilogue(alpha * op(A[b % nA]) * op(B[b % nB]) + beta * C[b])
//
// The instruction's rate bounds it: 128 flop per cycle and SM (37 TFLOP/s measured with every shape of it and with DFMA).
// What kept the block kernel at half of that was its own issue: eight warps that copied, met at a barrier and multiplied
// in step left the unit idle while they copied, and two such CTAs per SM hid that only where a third did not run alone.
// Here four warps do nothing but copy (cp.async into a ring, an mbarrier per stage each way) and eight do nothing but
// read fragments and multiply; one CTA per SM walks over the tiles, so that the ring runs on into the next tile while the
// last one is stored.  The reads are what is left beside the products (without any copies a product took 43 of 48 us), so
// they are 16 bytes wide: which k of a slab meet in a step, and which rows and columns of C a lane holds, is free as long as
// both operands and the stores agree.
//
// An operand stays as it lies in memory: slabs are [row][k] where k is contiguous and [k][row] where the rows are, lanes
// of a copy along the contiguous dimension (8-byte copies: an odd leading dimension aligns every other row only).
//   [row][k]  a lane reads k = 2 q, 2 q + 1 of rows r and r + 8 (q = lane % 4, r = lane / 4); rows 8 mod 16 doubles apart
//   [k][row]  a lane reads rows 2 r, 2 r + 1 at k = 2 q, and again at 2 q + 1; k rows 2 mod 8 doubles apart
// -- either way the eight lanes of a quarter warp lie in different banks.  4 x 500x389x640 with its backward pass: 189 us on the
// block kernel, 155 like this (its three products 45, 51 and 46; the tensor instruction alone would take 31 each).
#pragma once

#include "gemm_block.cuh"
#include "gemm_tc.cuh"

namespace zg {
namespace f64 {

constexpr int kLoaders = 128, kMath = 256, kThreads = kLoaders + kMath;
constexpr int TM = 64, TK = 32;
constexpr int kPitchK = TK + 8;

// 4 x 2 warps of 16 x (TN / 2) outputs
template <int TN, bool A_K, bool B_K>
struct Layout {
  static constexpr int kA = A_K ? TM * kPitchK : TK * (TM + 2), kB = B_K ? TN * kPitchK : TK * (TN + 2);
  static constexpr int kStage = kA + kB;  // doubles
  static constexpr int kFit = 226 * 1024 / (kStage * 8), kStages = kFit < 6 ? kFit : 6;
  static constexpr size_t kSmem = (size_t)kStages * kStage * sizeof(double);
};

struct Params {
  uint64_t nA, nB, m, n, k, lda, ldb, ldc, a_stride, b_stride, c_stride;
  double alpha, beta;
  const float* bias;
  const double* mask;
  uint32_t tiles_m, tiles_n, tiles;
  int epilogue;
  int* error_flag;
};

// D (16 x 8) += A (16 x 8) * B (8 x 8): lane l holds A[l / 4 (+ 8)][l % 4 (+ 4)] in a0 (a1; a2, a3), B[l % 4 (+ 4)][l / 4] and
// D[l / 4 (+ 8)][2 (l % 4), + 1]
__device__ __forceinline__ void mma(double (&d)[4], const double (&a)[4], double b0, double b1) {
  asm volatile("mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+d"(d[0]), "+d"(d[1]), "+d"(d[2]), "+d"(d[3]) : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(b0), "d"(b1));
}

// ROWS x TK elements of one operand into a stage, by the four loader warps; what lies outside is filled with zeros.
template <int ROWS, bool K_CONTIG>
__device__ __forceinline__ void copy_slab(double* dst, const double* src, uint64_t ld, uint64_t row0, uint64_t rows, uint64_t k0, uint64_t k) {
  constexpr int W = kLoaders / 32;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if constexpr (K_CONTIG) {
    const bool k_ok = k0 + lane < k;
    const int left = rows - row0 < (uint64_t)ROWS ? (int)(rows - row0) : ROWS;
    const double* s = src + (row0 + w) * ld + k0 + lane;
    double* d = dst + w * kPitchK + lane;
#pragma unroll
    for (int i = 0; i < ROWS / W; ++i) {
      const bool ok = k_ok && w + W * i < left;
      block::copy_async<8>(d + W * i * kPitchK, ok ? s : src, ok);
      s += W * ld;
    }
  } else {
    // 32 rows at a time; of 48, the second half warp of the odd pieces has nothing to do
    constexpr int P = (ROWS + 31) / 32, PITCH = ROWS + 2;
    const int left = k - k0 < (uint64_t)TK ? (int)(k - k0) : TK;
    const double* s = src + (k0 + w) * ld + row0 + lane;
    double* d = dst + w * PITCH + lane;
#pragma unroll
    for (int i = 0; i < TK / W; ++i) {
#pragma unroll
      for (int q = 0; q < P; ++q) {
        if (32 * q + 32 > ROWS && lane >= ROWS - 32 * q) continue;
        const bool ok = w + W * i < left && row0 + 32 * q + lane < rows;
        block::copy_async<8>(d + W * i * PITCH + 32 * q, ok ? s + 32 * q : src, ok);
      }
      s += W * ld;
    }
  }
}

template <int TN, bool A_K, bool B_K>
__global__ void __launch_bounds__(kThreads, 1) gemm_f64_kernel(const double* __restrict__ A, const double* __restrict__ B, double* C, const Params p) {
  using L = Layout<TN, A_K, B_K>;
  constexpr int S = L::kStages, NB = TN / 16;
  extern __shared__ __align__(16) double ring[];
  __shared__ uint64_t full[S], empty[S];
  __shared__ volatile int failed;
  if (threadIdx.x == 0) {
    failed = 0;
    for (int s = 0; s < S; ++s) {
      tc::mbar_init(&full[s], kLoaders);
      tc::mbar_init(&empty[s], kMath / 32);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  pdl_sync();
  const int slabs = (int)((p.k + TK - 1) / TK);
  uint32_t it = 0;  // slabs so far, over all tiles of this CTA
  auto place = [&](uint32_t tile, uint64_t& m0, uint64_t& n0) {
    n0 = (uint64_t)(tile % p.tiles_n) * TN;
    tile /= p.tiles_n;
    m0 = (uint64_t)(tile % p.tiles_m) * TM;
    return (uint64_t)(tile / p.tiles_m);
  };
  if (threadIdx.x < kLoaders) {
    bool go = true;
    for (uint32_t tile = blockIdx.x; tile < p.tiles && go; tile += gridDim.x) {
      uint64_t m0, n0;
      const uint64_t batch = place(tile, m0, n0);
      const double* a = A + batch % p.nA * p.a_stride;
      const double* b = B + batch % p.nB * p.b_stride;
      for (int c = 0; c < slabs; ++c, ++it) {
        const uint32_t s = it % S, round = it / S;
        if (round > 0 && !tc::mbar_wait(&empty[s], (round & 1) ^ 1, &failed)) { go = false; break; }
        double* as = ring + s * L::kStage;
        copy_slab<TM, A_K>(as, a, p.lda, m0, p.m, (uint64_t)c * TK, p.k);
        copy_slab<TN, B_K>(as + L::kA, b, p.ldb, n0, p.n, (uint64_t)c * TK, p.k);
        asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(tc::smem_u32(&full[s])) : "memory");
      }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
  } else {
    const int w = (threadIdx.x - kLoaders) >> 5, lane = threadIdx.x & 31, r = lane >> 2, q = lane & 3;
    const int wm = (w >> 1) * 16, wn = (w & 1) * (TN / 2);
    constexpr int pa = TM + 2, pb = TN + 2;
    const int a_at = A_K ? (wm + r) * kPitchK + 2 * q : 2 * q * pa + wm + 2 * r;
    const int b_at = L::kA + (B_K ? (wn + r) * kPitchK + 2 * q : 2 * q * pb + wn + 2 * r);
    // where D's rows (h) and block j's columns (e) lie in C's tile
    auto row_of = [&](int h) { return wm + (A_K ? r + 8 * h : 2 * r + h); };
    auto col_of = [&](int j, int e) {
      if (B_K || (NB % 2 && j == NB - 1)) return wn + 8 * j + 2 * q + e;
      return wn + 16 * (j / 2) + 2 * (2 * q + e) + (j & 1);
    };
    bool go = true;
    for (uint32_t tile = blockIdx.x; tile < p.tiles && go; tile += gridDim.x) {
      double acc[NB][4];
#pragma unroll
      for (int j = 0; j < NB; ++j) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.0;
      uint64_t m0, n0;
      const uint64_t batch = place(tile, m0, n0);
      double* c = C + batch * p.c_stride;
      const double* mk = p.mask ? p.mask + batch * p.c_stride : nullptr;
      const bool masked = p.epilogue == ZG_EPI_RELU_MASK, biased = p.epilogue == ZG_EPI_BIAS || p.epilogue == ZG_EPI_BIAS_RELU;
      // C and the mask are requested during the last slab, all in flight together: one by one behind it the 8 to 16 elements
      // of a thread are as many round trips
      double old[NB][4];
      unsigned off = 0;  // elements that the mask clears
      auto request = [&]() {
#pragma unroll
        for (int j = 0; j < NB; ++j)
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const uint64_t y = m0 + row_of(e >> 1), x = n0 + col_of(j, e & 1);
            const bool in = y < p.m && x < p.n;
            old[j][e] = in && p.beta != 0.0 ? c[y * p.ldc + x] : 0.0;
            if (masked && in && mk[y * p.ldc + x] <= 0.0) off |= 1u << (4 * j + e);
          }
      };
      if (slabs == 0) request();
      // Fragments are read one step (eight k) ahead of their products, over the slab's end as well: a warp that finished a slab
      // before it waited for the next one left the unit idle for some 340 cycles of 1536.
      struct Frag { double a[4], b[NB][2]; };
      Frag f[2];
      const double* st = ring;
      auto pair = [&](double& x, double& y, int at) {
        const double2 v = *reinterpret_cast<const double2*>(st + at);
        x = v.x;
        y = v.y;
      };
      auto read = [&](Frag& x, int kk) {
        if constexpr (A_K) {
          pair(x.a[0], x.a[2], a_at + kk);
          pair(x.a[1], x.a[3], a_at + 8 * kPitchK + kk);
        } else {
          pair(x.a[0], x.a[1], a_at + kk * pa);
          pair(x.a[2], x.a[3], a_at + (kk + 1) * pa);
        }
#pragma unroll
        for (int j = 0; j < NB; ++j) {
          if constexpr (B_K) {
            pair(x.b[j][0], x.b[j][1], b_at + 8 * j * kPitchK + kk);
          } else if (NB % 2 && j == NB - 1) {  // a block of its own: column r
            x.b[j][0] = st[b_at + 8 * j - r + kk * pb];
            x.b[j][1] = st[b_at + 8 * j - r + (kk + 1) * pb];
          } else if (j % 2 == 0) {
            pair(x.b[j][0], x.b[j + 1 < NB ? j + 1 : j][0], b_at + 8 * j + kk * pb);
            pair(x.b[j][1], x.b[j + 1 < NB ? j + 1 : j][1], b_at + 8 * j + (kk + 1) * pb);
          }
        }
      };
      auto multiply = [&](const Frag& x) {
#pragma unroll
        for (int j = 0; j < NB; ++j) mma(acc[j], x.a, x.b[j][0], x.b[j][1]);
      };
      auto enter = [&]() {  // slab `it`, and its first fragments
        const bool got = tc::mbar_wait(&full[it % S], it / S & 1, &failed);
        if (!__all_sync(0xffffffffu, got)) { go = false; return; }
        st = ring + it % S * L::kStage;
        read(f[0], 0);
      };
      auto leave = [&]() {  // all of slab `it` is in registers
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(&empty[it % S]);
        ++it;
      };
      if (slabs > 0) enter();
      for (int i = 0; i + 1 < slabs && go; ++i) {
#pragma unroll
        for (int t = 0; t < TK / 8; ++t) {
          if (t + 1 < TK / 8) read(f[(t + 1) & 1], 8 * (t + 1));
          else {
            leave();
            enter();
          }
          multiply(f[t & 1]);
        }
      }
      if (slabs > 0 && go) {
        const int steps = ((int)(p.k - (uint64_t)(slabs - 1) * TK) + 7) / 8;  // (a slab is padded with zeros)
        request();
#pragma unroll
        for (int t = 0; t < TK / 8; ++t) {
          if (t >= steps) break;
          if (t + 1 < steps) read(f[(t + 1) & 1], 8 * (t + 1));
          multiply(f[t & 1]);
        }
        leave();
      }
      if (!go) break;
#pragma unroll
      for (int j = 0; j < NB; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const uint64_t y = m0 + row_of(e >> 1), x = n0 + col_of(j, e & 1);
          if (y >= p.m || x >= p.n) continue;
          double v = p.alpha * acc[j][e];
          if (p.beta != 0.0) v += p.beta * old[j][e];
          if (biased) v += (double)p.bias[x];
          if (p.epilogue == ZG_EPI_BIAS_RELU) v = v > 0.0 ? v : 0.0;
          if (off >> (4 * j + e) & 1) v = 0.0;
          c[y * p.ldc + x] = v;
        }
    }
  }
  __syncthreads();
  if (threadIdx.x == 0 && failed && p.error_flag) *p.error_flag = 1;
}

}  // namespace f64
}  // namespace zg

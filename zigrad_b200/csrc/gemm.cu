// GEMM entry points: zg_bmm (include/zg_b200.h), gemm / gemv / ger
// (include/blas_conflux.h).  Large, TMA-addressable problems go to the
// tcgen05 kernel (gemm_tc.cuh); everything else (small shapes, rows whose byte
// stride is not a multiple of 16, fp64) runs on the FFMA kernel of gemm_block.cuh.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>

#include "common.cuh"
#include "driver_api.h"
#include "gemm_tc.cuh"
#include "gemm_tc_persistent.cuh"
#include "mlp_forward.cuh"
#include "gemm_skinny.cuh"
#include "gemm_block.cuh"
#include "gemm_f64.cuh"
#include "gemm_repack.cuh"
#include "mlp_tail.cuh"
#include "mlp_tail_rows.cuh"
#include "../../include/blas_conflux.h"

namespace zg {

static int g_math_mode = ZG_MATH_FP32X3;

// C[b][i][j] *= beta over an [m, n] window with leading dimension ldc
template <typename T>
__global__ void scale_c_kernel(T* C, size_t batches, size_t m, size_t n, size_t ldc, size_t c_stride, T beta) {
  pdl_sync();
  const size_t total = batches * m * n, nth = (size_t)gridDim.x * blockDim.x;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += nth) {
    const size_t b = i / (m * n), r = (i % (m * n)) / n, cidx = i % n;
    T* p = C + b * c_stride + r * ldc + cidx;
    *p = (beta == T(0)) ? T(0) : beta * (*p);
  }
}

template <typename T>
static void prescale_c(cudaStream_t s, T* C, size_t batches, size_t m, size_t n, size_t ldc, size_t c_stride, double beta) {
  if (beta == 1.0) return;
  launch_pdl(scale_c_kernel<T>, dim3(grid_for(batches * m * n, 1024)), dim3(256), 0, s, C, batches, m, n, ldc, c_stride, (T)beta);
}

// The tiles of the persistent kernel's list from `whole` on, cleared for the K ranges that are added into them: 9 MB of the
// 67 MB of a 4096 x 4096 product.  Grid: (row strips of 32, tiles); n is a multiple of four.
__global__ void __launch_bounds__(256) clear_tiles_kernel(float* C, uint32_t m, uint32_t n, size_t ldc, size_t c_stride, uint32_t tiles_m, uint32_t tiles_n, uint32_t whole) {
  pdl_sync();
  const tc::TileCoord t = tc::tile_coord(whole + blockIdx.y, tiles_m, tiles_n, 0xffffffffu, 1);
  const uint32_t col = t.n * tc::kPBN + threadIdx.x % 64 * 4;
  if (col >= n) return;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const uint32_t row = t.m * tc::kPBM + blockIdx.x * 32 + threadIdx.x / 64 + 4 * i;
    if (row < m) *reinterpret_cast<float4*>(C + t.batch * c_stride + row * ldc + col) = make_float4(0.f, 0.f, 0.f, 0.f);
  }
}

// Cluster size of a small problem: enough CTAs to occupy the SMs, no k range under 32.
static unsigned block_splits(size_t tiles, len_t k) {
  unsigned s = 1;
  while (s < 8 && tiles * s * 2 <= (size_t)sm_count() * 2 && k >= (len_t)s * 2 * 32) s *= 2;
  return s;
}

template <typename TI, typename TC, int TM, int TN, int MI>
static void launch_block_inst(cudaStream_t s, const void* A, const void* B, void* C, block::Params& p, len_t nC, unsigned splits) {
  using L = block::Layout<TI, TM, TN, MI>;
  auto kern = block::gemm_block_kernel<TI, TC, TM, TN, MI>;
  static SharedMemoryLimit limit;
  if (!limit.raise(kern, L::kSmem)) return;
  p.tiles_m = (uint32_t)((p.m + TM - 1) / TM);
  p.tiles_n = (uint32_t)((p.n + TN - 1) / TN);
  p.splits = splits;
  p.k_per_split = splits > 1 ? ((p.k + splits - 1) / splits + 7) / 8 * 8 : p.k;
  const size_t ctas = (size_t)p.tiles_m * p.tiles_n * nC * splits;
  if (ctas > 0x7fffffffu) { set_error(kBadArgument, "gemm: grid too large (m=%lu, batches=%lu)", (len_t)p.m, nC); return; }
  launch_pdl_cluster(kern, dim3((unsigned)ctas), dim3(block::kThreads), L::kSmem, s, splits, static_cast<const TI*>(A),
                     static_cast<const TI*>(B), static_cast<TC*>(C), p);
}

template <int TN, bool A_K, bool B_K>
static void launch_f64_inst(cudaStream_t s, const void* A, const void* B, void* C, const f64::Params& p) {
  using L = f64::Layout<TN, A_K, B_K>;
  auto kern = f64::gemm_f64_kernel<TN, A_K, B_K>;
  static SharedMemoryLimit limit;
  if (!limit.raise(kern, L::kSmem)) return;
  launch_pdl(kern, dim3(std::min<unsigned>(p.tiles, (unsigned)sm_count())), dim3(f64::kThreads), L::kSmem, s, static_cast<const double*>(A),
             static_cast<const double*>(B), static_cast<double*>(C), p);
}

static int* tc_error_flag();

// The tile width whose busiest SM has the least to do: the tensor instruction takes TN cycles per k of a 64 x TN tile, and a
// tile about 300 cycles beside.
static void launch_f64(cudaStream_t s, const void* A, const void* B, void* C, block::Params& q, len_t nC) {
  f64::Params p;
  memset(&p, 0, sizeof(p));
  p.nA = q.nA; p.nB = q.nB; p.m = q.m; p.n = q.n; p.k = q.k; p.lda = q.lda; p.ldb = q.ldb; p.ldc = q.ldc;
  p.a_stride = q.a_stride; p.b_stride = q.b_stride; p.c_stride = q.c_stride;
  p.alpha = q.alpha; p.beta = q.beta; p.bias = q.bias; p.mask = static_cast<const double*>(q.mask); p.epilogue = q.epilogue;
  p.error_flag = tc_error_flag();
  const size_t sms = (size_t)sm_count(), tiles_m = (p.m + f64::TM - 1) / f64::TM;
  size_t tn = 0;
  double best = 0;
  for (const size_t w : {64, 48, 32}) {
    const double tiles = (double)tiles_m * (double)((p.n + w - 1) / w) * (double)nC;
    const double cost = std::ceil(tiles / (double)sms) * ((double)w * (double)p.k + 300.0);
    if (!tn || cost < best) { tn = w; best = cost; }
  }
  const size_t tiles = tiles_m * ((p.n + tn - 1) / tn) * nC;
  // A slab or two per tile, and C only written: what counts is how many tiles an SM has in flight, and the block kernel has two
  // (us, it and the persistent one: 28 x 213x121x17 8.0 and 10.6, 6 x 476x348x44 10.0 and 12.9, 9 x 76x1596x20 13.8 and 16.8;
  // 2 x 632x551x20 8.2 and 8.5, 5 x 1144x635x8 22.3 and 22.6; with C read as well 950x419x6 19 and 9).  A tile per SM or little
  // more is a chain of copies, of which a [k][row] operand has more than the four copying warps issue in time (4 x 187x603x9
  // 5.0 and 6.8, 2 x 302x817x60 7.2 and 8.8, with a tile and a fifth per SM 5 x 215x479x14 6.8 and 8.0; with B in rows of k 4 x 672x174x65 8.8 and 7.8).
  const size_t t64 = tiles_m * ((p.n + 63) / 64) * nC, short_k = t64 * 5 > sms * 6 ? 48 : (q.tb ? 0 : (t64 > sms ? 24 : 80));
  if (p.n * 16 >= (p.n + 63) / 64 * (64 * 13) && p.beta == 0.0 && p.epilogue != ZG_EPI_RELU_MASK && p.k <= short_k) return launch_block_inst<double, double, 64, 64, 0>(s, A, B, C, q, nC, 1);
  if (tiles > 0x7fffffffu) { set_error(kBadArgument, "gemm: grid too large (m=%lu, batches=%lu)", (len_t)p.m, nC); return; }
  p.tiles_m = (uint32_t)tiles_m;
  p.tiles_n = (uint32_t)((p.n + tn - 1) / tn);
  p.tiles = (uint32_t)tiles;
#define ZG_F64_CASE(TNV)                                                             \
  if (tn == TNV) {                                                                   \
    if (!q.ta && q.tb) return launch_f64_inst<TNV, true, true>(s, A, B, C, p);       \
    if (!q.ta) return launch_f64_inst<TNV, true, false>(s, A, B, C, p);              \
    if (q.tb) return launch_f64_inst<TNV, false, true>(s, A, B, C, p);               \
    return launch_f64_inst<TNV, false, false>(s, A, B, C, p);                        \
  }
  ZG_F64_CASE(64)
  ZG_F64_CASE(48)
  ZG_F64_CASE(32)
#undef ZG_F64_CASE
}

template <typename TI, typename TC>
static void launch_block(cudaStream_t s, const void* A, const void* B, void* C, len_t nA, len_t nB, len_t nC, len_t m, len_t n, len_t k,
                         bool ta, bool tb, len_t lda, len_t ldb, len_t ldc, double alpha, double beta, int epilogue, const void* bias,
                         const void* mask, void* colsum) {
  block::Params p;
  memset(&p, 0, sizeof(p));
  p.nA = nA; p.nB = nB; p.m = m; p.n = n; p.k = k; p.lda = lda; p.ldb = ldb; p.ldc = ldc;
  p.a_stride = (ta ? k : m) * lda; p.b_stride = (tb ? n : k) * ldb; p.c_stride = m * ldc;
  p.ta = ta; p.tb = tb; p.alpha = alpha; p.beta = beta; p.epilogue = epilogue;
  p.bias = static_cast<const float*>(bias); p.mask = mask; p.colsum = static_cast<float*>(colsum);
  const size_t t64 = ((m + 63) / 64) * ((n + 63) / 64) * nC, t32 = ((m + 31) / 32) * ((n + 31) / 32) * nC;
  if constexpr (sizeof(TI) == 8) {
    // Half a 64 x 64 tile per SM or less: 32 x 32 tiles split over clusters.  (An fp64 caller has no column sums.)
    if (t64 * 2 <= (size_t)sm_count()) launch_block_inst<TI, TC, 32, 32, 0>(s, A, B, C, p, nC, block_splits(t32, k));
    else launch_f64(s, A, B, C, p, nC);
  } else {
    // 64 x 64 tiles (half the copies per multiply-add) once there is one for every SM; below that, parallelism counts
    // for more: 1000x301x501 takes 21 us with 32 x 32, 30 with 64 x 64; 4096x1023x1023 379 and 280
    if (t64 > (size_t)sm_count()) launch_block_inst<TI, TC, 64, 64, 8>(s, A, B, C, p, nC, 1);
    else launch_block_inst<TI, TC, 32, 32, 4>(s, A, B, C, p, nC, block_splits(t32, k));
  }
}

// =====================================================================
// tcgen05 path: host side
// =====================================================================
static int* tc_error_flag() {
  // one device-visible flag per device, read back by zg_last_error callers via check_tc_errors()
  static int* flags[64] = {nullptr};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return nullptr;
  if (!flags[dev]) {
    int* p = nullptr;
    if (cudaMalloc(&p, sizeof(int)) != cudaSuccess) { (void)cudaGetLastError(); return nullptr; }
    // the legacy stream does not order against the library's non-blocking streams: finish the clear here
    cudaMemset(p, 0, sizeof(int));
    cudaDeviceSynchronize();
    flags[dev] = p;
  }
  return flags[dev];
}

static bool make_tmap(CUtensorMap* map, bool bf16, const void* base, uint64_t inner, uint64_t rows, uint64_t batches, uint64_t ld,
                      uint32_t box_inner, uint32_t box_rows, bool atom32) {
  static auto encode = ZG_DRV(cuTensorMapEncodeTiled);
  if (!encode) return false;
  const uint64_t es = bf16 ? 2 : 4;
  cuuint64_t dims[3] = {inner, rows, batches};
  cuuint64_t strides[2] = {ld * es, rows * ld * es};
  cuuint32_t box[3] = {box_inner, box_rows, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = encode(map, bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<void*>(base), dims,
                      strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                      atom32 ? CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B : CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                      CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return ZG_CU(r);
}

template <int BN, bool AK, bool BK_, int MODE, bool DIRECT = false>
static bool launch_tc_inst(cudaStream_t s, const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& tcm, const tc::Params& p, dim3 grid) {
  using SL = tc::SmemLayout<BN, MODE>;
  auto kern = tc::gemm_tc_kernel<BN, AK, BK_, MODE, DIRECT>;
  static SharedMemoryLimit limit;
  if (!limit.raise(kern, SL::kTotal)) return false;
  return launch_pdl_cluster(kern, grid, dim3(SL::kThreads + (DIRECT ? tc::kLoadWarps * 32 : 0)), (size_t)SL::kTotal, s, p.cluster ? p.splits : 1, ta, tb, tcm, p);
}

template <int MODE>
static bool launch_tc_mode(cudaStream_t s, int bn, bool a_kmajor, bool b_kmajor, const CUtensorMap& ta, const CUtensorMap& tb,
                           const CUtensorMap& tcm, const tc::Params& p, dim3 grid) {
#define ZG_TC_CASE(BNV)                                                                       \
  if (bn == BNV) {                                                                            \
    if (a_kmajor && b_kmajor) return launch_tc_inst<BNV, true, true, MODE>(s, ta, tb, tcm, p, grid);   \
    if (a_kmajor && !b_kmajor) return launch_tc_inst<BNV, true, false, MODE>(s, ta, tb, tcm, p, grid); \
    if (!a_kmajor && b_kmajor) return launch_tc_inst<BNV, false, true, MODE>(s, ta, tb, tcm, p, grid); \
    return launch_tc_inst<BNV, false, false, MODE>(s, ta, tb, tcm, p, grid);                       \
  }
  if constexpr (!tc::ModeTraits<MODE>::kBf16) { ZG_TC_CASE(32) }
  ZG_TC_CASE(64)
  ZG_TC_CASE(128)
#undef ZG_TC_CASE
  set_error(kBadArgument, "gemm: no tensor-core instance for BN=%d", bn);
  return false;
}

static void launch_tc_direct(cudaStream_t s, int bn, bool a_kmajor, bool b_kmajor, const CUtensorMap& ta, const CUtensorMap& tb,
                             const CUtensorMap& tcm, const tc::Params& p, dim3 grid) {
#define ZG_DIRECT_CASE(BNV)                                                                                        \
  if (a_kmajor && b_kmajor) launch_tc_inst<BNV, true, true, tc::kFP32X3, true>(s, ta, tb, tcm, p, grid);     \
  else if (a_kmajor) launch_tc_inst<BNV, true, false, tc::kFP32X3, true>(s, ta, tb, tcm, p, grid);           \
  else if (b_kmajor) launch_tc_inst<BNV, false, true, tc::kFP32X3, true>(s, ta, tb, tcm, p, grid);           \
  else launch_tc_inst<BNV, false, false, tc::kFP32X3, true>(s, ta, tb, tcm, p, grid);
  if (bn == 64) { ZG_DIRECT_CASE(64) } else { ZG_DIRECT_CASE(128) }
#undef ZG_DIRECT_CASE
}

// Clusters of `size` CTAs that can run at once when a CTA takes a whole SM (GPCs hold different numbers of SMs, so not
// every SM finds a place: of 148, 148 CTAs in pairs, 132 in fours and sixes, 120 in eights).
static size_t max_clusters(unsigned size) {
  static int cached[9] = {0};
  if (!cached[size]) {
    using SL = tc::SmemLayout<64, tc::kFP32X3>;
    auto kern = tc::gemm_tc_kernel<64, true, true, tc::kFP32X3>;
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3(size);
    cfg.blockDim = dim3(SL::kThreads);
    cfg.dynamicSmemBytes = SL::kTotal;
    cudaLaunchAttribute attr;
    memset(&attr, 0, sizeof(attr));
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = size;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (!ZG_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SL::kTotal)) ||
        !ZG_CUDA(cudaOccupancyMaxActiveClusters(&n, kern, &cfg)))
      return 0;
    cached[size] = n + 1;  // 0: not asked yet
  }
  return (size_t)(cached[size] - 1);
}

template <bool AK, bool BK_, int MODE>
static bool launch_persistent_inst(cudaStream_t s, const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& tcm, const CUtensorMap& tmm,
                                   const tc::Params& p, uint32_t tiles_m,
                                   uint32_t tiles_n, uint32_t n_tiles) {
  using SL = tc::PersistentSmem<MODE>;
  auto kern = tc::gemm_tc_persistent_kernel<AK, BK_, MODE>;
  static SharedMemoryLimit limit;
  if (!limit.raise(kern, SL::kTotal)) return false;
  const unsigned pairs = std::min<unsigned>(n_tiles, (unsigned)sm_count() / 2);
  // work-item counter: zero between launches (slot 2 of the stream's workspace)
  unsigned* unused = nullptr;
  unsigned* counter = static_cast<unsigned*>(workspace(s, 256, &unused, 2));
  if (!counter) return false;
  return launch_pdl_cluster(kern, dim3(2 * pairs), dim3(tc::kThreadsPersistent), (size_t)SL::kTotal, s, 2u, ta, tb, tcm, tmm, p, tiles_m, tiles_n, n_tiles, counter);
}

template <int MODE>
static bool launch_persistent(cudaStream_t s, bool a_kmajor, bool b_kmajor, const CUtensorMap& ta, const CUtensorMap& tb,
                              const CUtensorMap& tcm, const CUtensorMap& tmm, const tc::Params& p, uint32_t tiles_m, uint32_t tiles_n, uint32_t n_tiles) {
  if (a_kmajor && b_kmajor) return launch_persistent_inst<true, true, MODE>(s, ta, tb, tcm, tmm, p, tiles_m, tiles_n, n_tiles);
  if (a_kmajor && !b_kmajor) return launch_persistent_inst<true, false, MODE>(s, ta, tb, tcm, tmm, p, tiles_m, tiles_n, n_tiles);
  if (!a_kmajor && b_kmajor) return launch_persistent_inst<false, true, MODE>(s, ta, tb, tcm, tmm, p, tiles_m, tiles_n, n_tiles);
  return launch_persistent_inst<false, false, MODE>(s, ta, tb, tcm, tmm, p, tiles_m, tiles_n, n_tiles);
}

// fp32 problems with n <= 16 or k <= 16 (see gemm_skinny.cuh).  Returns true when taken.
static bool try_skinny(dtype id, dtype c_id, cudaStream_t s, const void* A, const void* B, void* C, len_t nA, len_t nB, len_t nC, len_t m,
                       len_t n, len_t k, bool ta, bool tb, len_t lda, len_t ldb, len_t ldc, double alpha, double beta, int epilogue,
                       const void* bias, const void* mask, void* colsum) {
  static const bool off = [] { const char* e = getenv("ZG_GEMM_NO_SKINNY"); return e && e[0] == '1'; }();
  if (off || id != SINGLE || c_id != SINGLE || nA != 1 || nB != 1 || nC != 1) return false;
  if (m > 0x7fffffffu || k == 0 || k > 0x7fffffffu || lda > 0xffffffffu || ldb > 0xffffffffu || ldc > 0xffffffffu) return false;
  skinny::Params p;
  p.A = static_cast<const float*>(A); p.B = static_cast<const float*>(B); p.C = static_cast<float*>(C);
  p.bias = static_cast<const float*>(bias); p.mask = static_cast<const float*>(mask); p.colsum = static_cast<float*>(colsum);
  p.m = (uint32_t)m; p.n = (uint32_t)n; p.k = (uint32_t)k;
  p.lda = (uint32_t)lda; p.ldb = (uint32_t)ldb; p.ldc = (uint32_t)ldc;
  p.alpha = (float)alpha; p.beta = (float)beta; p.epilogue = epilogue; p.tb = tb ? 1 : 0;
  if (ta) {
    // weight gradient of a narrow layer: A [k, m], B [k, n]
    if (tb || m > 16 || n < 16 || n > 256 || 256 % n != 0 || k < 1024 || epilogue != ZG_EPI_NONE || colsum) return false;
    prescale_c<float>(s, static_cast<float*>(C), 1, m, n, ldc, m * ldc, beta);
    const size_t ctas = std::min<size_t>((k + 31) / 32, (size_t)sm_count() * 2);
    const uint32_t rows_per_cta = (uint32_t)((k + ctas - 1) / ctas);
    const unsigned grid = (unsigned)((k + rows_per_cta - 1) / rows_per_cta);
    const int mmax = m <= 4 ? 4 : (m <= 8 ? 8 : (m <= 12 ? 12 : 16));
    const size_t smem = (size_t)(skinny::kThreads / n) * mmax * n * sizeof(float);
    if (mmax == 4) return launch_pdl(skinny::skinny_m_kernel<4>, dim3(grid), dim3(skinny::kThreads), smem, s, p, rows_per_cta);
    if (mmax == 8) return launch_pdl(skinny::skinny_m_kernel<8>, dim3(grid), dim3(skinny::kThreads), smem, s, p, rows_per_cta);
    if (mmax == 12) return launch_pdl(skinny::skinny_m_kernel<12>, dim3(grid), dim3(skinny::kThreads), smem, s, p, rows_per_cta);
    return launch_pdl(skinny::skinny_m_kernel<16>, dim3(grid), dim3(skinny::kThreads), smem, s, p, rows_per_cta);
  }
  if (m < 256) return false;
  // (deeper rows: the quad per row walks them serially, 37 us for 20000x16x500 against 10 on the tensor cores)
  if (n <= 16 && k >= 16 && k <= 128 && k % 4 == 0 && lda % 4 == 0 && host_aligned16(A) && epilogue != ZG_EPI_RELU_MASK && !colsum) {
    const unsigned grid = (unsigned)((m + skinny::kThreads / 4 - 1) / (skinny::kThreads / 4));
    const size_t smem = (size_t)n * k * sizeof(float);
    if (n <= 4) return launch_pdl(skinny::skinny_n_kernel<4>, dim3(grid), dim3(skinny::kThreads), smem, s, p);
    if (n <= 8) return launch_pdl(skinny::skinny_n_kernel<8>, dim3(grid), dim3(skinny::kThreads), smem, s, p);
    if (n <= 12) return launch_pdl(skinny::skinny_n_kernel<12>, dim3(grid), dim3(skinny::kThreads), smem, s, p);
    return launch_pdl(skinny::skinny_n_kernel<16>, dim3(grid), dim3(skinny::kThreads), smem, s, p);
  }
  if (k <= 16 && n >= 16 && n <= 256 && n % 4 == 0 && ldc % 4 == 0 && host_aligned16(C) && beta == 0.0 &&
      (epilogue != ZG_EPI_RELU_MASK || host_aligned16(mask)) && (!bias || host_aligned16(bias))) {
    const size_t cg = n / 4;
    if (colsum && (cg & (cg - 1)) != 0) return false;  // a thread keeps one column group only when cg divides the stride
    const size_t want = (m * cg + skinny::kThreads - 1) / skinny::kThreads;
    const unsigned grid = (unsigned)std::min<size_t>(want, (size_t)sm_count() * 8);
    const size_t smem = ((size_t)n * k + n) * sizeof(float);
    if (k <= 4) return launch_pdl(skinny::skinny_k_kernel<4>, dim3(grid), dim3(skinny::kThreads), smem, s, p);
    if (k <= 8) return launch_pdl(skinny::skinny_k_kernel<8>, dim3(grid), dim3(skinny::kThreads), smem, s, p);
    if (k <= 12) return launch_pdl(skinny::skinny_k_kernel<12>, dim3(grid), dim3(skinny::kThreads), smem, s, p);
    return launch_pdl(skinny::skinny_k_kernel<16>, dim3(grid), dim3(skinny::kThreads), smem, s, p);
  }
  return false;
}

// SM budget of the zg_bmm call in progress (zg_bmm_sm_budget): GEMMs that run side by side on parallel
// streams size their split-K grids for a share of the SMs, so that together they fit in one wave
// (a CTA of these kernels takes a whole SM's shared memory; an oversubscribed launch runs its
// surplus CTAs in a second wave after the first has drained).
static thread_local int g_next_sm_budget = 0, g_sm_budget = 0;
static size_t sm_share() {
  const size_t all = (size_t)sm_count();
  return (g_sm_budget > 0 && (size_t)g_sm_budget < all) ? (size_t)g_sm_budget : all;
}
// bf16 operands with 16-byte rows into an fp32 C whose sums shall round all the same (zg_bmm_rounded_sums)
static thread_local bool g_next_rounded = false, g_rounded = false;
extern "C" void zg_bmm_rounded_sums(int on) { g_next_rounded = on != 0; }
extern "C" void zg_bmm_sm_budget(int sms) { g_next_sm_budget = sms > 0 ? sms : 0; }

// Operands without 16-byte rows copied with them (gemm_repack.cuh) into the stream's buffer for that; a pointer and leading
// dimension are replaced where they are copied.  False: no place for them (more than 256 MB, or copy_space() has none).
template <typename T>
static bool repack_operands(cudaStream_t s, const void*& A, uint64_t rows_a, uint64_t cols_a, len_t& lda, bool copy_a, const void*& B, uint64_t rows_b,
                            uint64_t cols_b, len_t& ldb, bool copy_b, std::unique_lock<std::mutex>& held) {
  constexpr uint64_t E = 16 / sizeof(T);
  auto words = [](uint64_t cols) { return (cols + E - 1) / E; };
  const uint64_t wa = copy_a ? rows_a * words(cols_a) : 0, wb = copy_b ? rows_b * words(cols_b) : 0;
  const uint64_t at_b = (wa * 16 + 255) / 256 * 256, bytes = at_b + wb * 16;
  char* ws = bytes > ((uint64_t)256 << 20) ? nullptr : static_cast<char*>(copy_space(s, bytes, held));
  if (!ws) return false;
  const repack::Operand a{A, ws, lda, (uint32_t)cols_a, (uint32_t)words(cols_a), wa}, b{B, ws + at_b, ldb, (uint32_t)cols_b, (uint32_t)words(cols_b), wb};
  const unsigned grid = grid_for(std::max(wa, wb), 512);
  if (!launch_pdl(repack::repack_kernel<T>, dim3(grid, copy_a && copy_b ? 2 : 1), dim3(256), 0, s, copy_a ? a : b, b)) return false;
  if (copy_a) { A = a.dst; lda = words(cols_a) * E; }
  if (copy_b) { B = b.dst; ldb = words(cols_b) * E; }
  return true;
}

// Returns true when the tensor-core path took the problem.
static bool try_tensor_core(dtype id, dtype c_id, cudaStream_t s, const void* A, const void* B, void* C, len_t nA, len_t nB, len_t nC,
                            len_t m, len_t n, len_t k, bool ta, bool tb, len_t lda, len_t ldb, len_t ldc, double alpha, double beta,
                            int epilogue, const void* bias, const void* mask, void* colsum) {
  const bool bf16 = (id == BF16);
  if (!(id == SINGLE || bf16)) return false;
  if (id == SINGLE && (g_math_mode == ZG_MATH_FFMA || c_id != SINGLE)) return false;
  if (bf16 && !(c_id == SINGLE || c_id == BF16)) return false;
  const size_t es = bf16 ? 2 : 4;
  // operands whose rows a TMA box cannot address: fp32 ones are copied element by element (direct_slab)
  bool a_direct = !host_aligned16(A) || (lda * es) % 16 != 0, b_direct = !host_aligned16(B) || (ldb * es) % 16 != 0;
  bool direct = a_direct || b_direct;
  if (m == 0 || n == 0 || nC == 0) return false;
  if (m > 0x7fffffffu || n > 0x7fffffffu || k > 0x7fffffffu || ldc > 0xffffffffu) return false;
  // Small problems are a latency chain on the tensor cores (descriptor fetch, TMA round trip, operand split, MMA,
  // TMEM read-back: 7 to 9 us in three passes, 4 in one); the FFMA kernel with its clusters needs 3 us + 1 us per 9.5 M
  // multiply-adds.  Measured crossovers: 50 M in three passes (512x128x784: 8.5 us either way; 64x128x784 4.1
  // against 13.8), 4 M in one (bf16 64x128x784 = 6.4 M: 6.0 against 5.6).
  const int mode = bf16 ? tc::kBF16 : (g_math_mode == ZG_MATH_TF32 && !direct ? tc::kTF32 : tc::kFP32X3);
  const double small = mode == tc::kFP32X3 ? 5e7 : 4e6;
  static const bool force = [] { const char* e = getenv("ZG_GEMM_FORCE_TC"); return e && e[0] == '1'; }();
  const double macs = (double)((m + 31) / 32 * 32) * (double)((n + 31) / 32 * 32) * (double)k * (double)nC;  // its tiles are 32 x 32
  if (!force && macs < small) return false;
  // A bf16 product of such operands with an fp32 C went to the FFMA kernel, whose sums round to nearest; on the tensor cores
  // it takes the form that adds up as exactly (kBF16Sums).  128-wide tiles without a carry from k = 640 on where the FFMA kernel
  // has no K ranges: 0.96 to 0.15 of that kernel's error there; 64-wide ones with it 1.0 to 0.15 from k = 96 on (below that
  // 1.1 to 1.3, and the FFMA kernel stays): 130 random shapes up to k = 8000.  2309x3283x565 382 us and 94 like this, 1208x1518x782
  // 158 and 16; 331x17x2571 12.6 and 13.6.
  // Measured crossovers of the copy: bf16 with a bf16 C against the FFMA kernel 10 M multiply-adds (8.0 us either way; 30 M: 17 and 9).  fp32
  // against the element-wise ring, which fetches an operand once for every 128 rows or columns of C: from two and a half
  // times the words of the copy on, and 5 M in all, 15 M with few slabs per tile (160 random shapes: within 1.1 % of the better
  // of the two, a rule on the multiply-adds 10 %; 468x230x4071 24 and 18 us, 2248x593x5015 138 and 95, 1613x1194x239 13.7 and
  // 14.6, 100x4097x4097 33 and 51).
  const double words_a = a_direct ? (double)nA * (double)m * (double)k : 0.0, words_b = b_direct ? (double)nB * (double)n * (double)k : 0.0;
  const double fetched = (words_a ? (double)nC * (double)m * (double)k : 0.0) * (double)((n + 127) / 128) +
                         (words_b ? (double)nC * (double)n * (double)k : 0.0) * (double)((m + 127) / 128);
  const bool copies_pay = fetched >= 2.5 * (words_a + words_b) && fetched >= (k >= 512 ? 5e6 : 1.5e7);
  const bool sums = bf16 && (direct || g_rounded) && c_id == SINGLE;
  if (sums && (macs < 2e7 || k < 96)) return false;
  std::unique_lock<std::mutex> copies;  // until the product has been launched
  if (direct && (bf16 ? macs >= 1.5e7 : copies_pay)) {
    const uint64_t ra = nA * (ta ? k : m), ca = ta ? m : k, rb = nB * (tb ? n : k), cb = tb ? k : n;
    if (bf16 ? repack_operands<__nv_bfloat16>(s, A, ra, ca, lda, a_direct, B, rb, cb, ldb, b_direct, copies)
             : repack_operands<float>(s, A, ra, ca, lda, a_direct, B, rb, cb, ldb, b_direct, copies))
      a_direct = b_direct = direct = false;
  }
  if (direct && bf16) return false;
  const int atom = bf16 ? 64 : 32;        // M/N elements per 128-byte column block
  const int bk = bf16 ? 64 : 32;
  // A C of few rows is computed as its transpose, so that the long dimension fills the 128 rows of the tile.
  // (Only where the column tiles alone occupy the chip in clusters of eight.)
  const bool swap = m <= 64 && n >= 1536;
  const len_t M = swap ? n : m, N = swap ? m : n;
  const bool a_kmajor = swap ? tb : !ta;  // the dimension that is contiguous in memory: K, or M / N
  const bool b_kmajor = swap ? !ta : tb;
  // Large single-pass problems: persistent kernel over 256 x 256 tiles of CTA pairs
  // (a tile for half of them at least, k deep enough to amortise the tile hand-over).
  static const bool no_persist = [] { const char* e = getenv("ZG_GEMM_NO_PERSISTENT"); return e && e[0] == '1'; }();
  const size_t ptiles = ((m + tc::kPBM - 1) / tc::kPBM) * ((n + tc::kPBN - 1) / tc::kPBN) * nC, pairs = (size_t)sm_count() / 2;
  const bool persistent = mode != tc::kFP32X3 && !sums && !swap && n > 128 && k >= 8 * (size_t)bk && ptiles * 2 >= pairs &&
                          ptiles <= 0x3fffffffu && !no_persist;
  int bn = persistent ? 256 : (N <= 32 && !direct ? 32 : (N <= 64 ? 64 : 128));
  if (sums) bn = k >= 640 && N > 64 && block_splits(((m + 31) / 32) * ((n + 31) / 32) * nC, k) == 1 ? 128 : 64;
  if (bn < atom) bn = atom;               // MN-major B needs whole column blocks; bf16 has no BN=32 instance
  size_t tiles = ((M + 127) / 128) * ((N + bn - 1) / bn) * nC;
  // Problems with few tiles get their parallelism from K splits.  Up to eight splits form a cluster, which sums its
  // partial tiles through distributed shared memory and applies any epilogue.  A plain product of 128-wide tiles
  // adds them into C with TMA reductions instead (128x784x1024: 7.2 us against 8.8), which also allows more
  // than eight.  What cannot split, or only in two, halves BN when there are too few tiles to occupy the SMs
  // (8192x128x784: 12.6 us in 64-wide tiles, 14.4 as two splits of 128-wide ones).
  bool c_aligned;
  {
    const size_t ce = (c_id == SINGLE) ? 4 : 2;
    c_aligned = host_aligned16(C) && (ldc * ce) % 16 == 0 && ((uint64_t)m * ldc * ce) % 16 == 0;
    if (mask) c_aligned = c_aligned && host_aligned16(mask);
    if (bias) c_aligned = c_aligned && host_aligned16(bias);
  }
  const size_t min_slabs = mode == tc::kFP32X3 || sums ? 4 : 12;  // per split: a three-pass slab costs 450 to 750 cycles, a single-pass one 130
  const bool can_split = !persistent && k >= 2 * min_slabs * (size_t)bk && tiles * (bn == 128 ? 3 : 2) <= sm_share();
  // (in a cluster; a plain product of 128-wide tiles reduces through the tensor map)
  auto cluster_splits = [&](size_t t) {
    unsigned sp = (unsigned)std::max<size_t>(1, std::min({sm_share() / t, (size_t)k / (min_slabs * bk), (size_t)8}));
    while (sp > 1 && t > max_clusters(sp)) --sp;
    return sp;
  };
  const bool reduces = epilogue == ZG_EPI_NONE && !colsum && c_id == SINGLE && c_aligned && !swap && bn == 128;
  const size_t tiles64 = ((M + 127) / 128) * ((N + 63) / 64) * nC;
  if (!persistent && !can_split && bn == 128 && !sums && tiles * 2 <= sm_share() && N > 64) {
    bn = 64;
    tiles = tiles64;
  } else if (can_split && mode == tc::kFP32X3 && bn == 128 && !reduces && tiles64 <= sm_share()) {
    // Three-pass tiles in clusters: a 128-wide one takes about 0.6 us per slab, 6.8 us beside it and 1.4 more in a cluster of
    // eight, a 64-wide one 0.37 and 5.8 (launch, first loads, staging, the cluster's sum).  1000x301x501 11.8 us in 128-wide
    // tiles, 9.8 in 64-wide ones; 4096x128x256 9.2 and 7.2; 1000x501x1000 12.3 and 12.5.
    // Where the ring copies element by element a slab takes about a microsecond in either (163x1429x1194 19.2 us in 64-wide
    // tiles of three ranges, 15.2 in 128-wide ones of six; 887x179x3198 19.3 and 21.7).
    auto slabs = [&](unsigned sp) { return (double)((k + (size_t)bk * sp - 1) / ((size_t)bk * sp)); };
    const unsigned s128 = cluster_splits(tiles), s64 = cluster_splits(tiles64);
    if (direct ? 3.2 + 0.95 * slabs(s64) < 8.0 + slabs(s128) : 5.8 + 0.37 * slabs(s64) < 6.8 + 0.6 * slabs(s128) + (s128 == 8 ? 1.4 : 0.0)) {
      bn = 64;
      tiles = tiles64;
    }
  }
  unsigned splits = 1;
  size_t whole = ptiles;
  if (persistent && epilogue == ZG_EPI_NONE && !colsum && c_id == SINGLE) {
    // The tiles of the last wave as K ranges, when those fill it better: its length in k-slabs, with two slabs' time for
    // what every item costs, over the numbers of ranges (at least 16 slabs each).
    const size_t rest = ptiles % pairs, slabs = (k + bk - 1) / bk;
    size_t best = slabs + 2;
    for (unsigned sp = 2; rest && sp <= 16 && slabs / sp >= 16; ++sp) {
      const size_t len = (rest * sp + pairs - 1) / pairs * ((slabs + sp - 1) / sp + 2);
      if (len + slabs / 32 < best) { best = len; splits = sp; }
    }
    if (splits > 1) whole = ptiles - rest;
  }
  bool cluster = false;
  if (can_split) {
    if (reduces) {
      splits = (unsigned)std::max<size_t>(1, std::min(sm_share() / tiles, k / (min_slabs * bk)));
    } else {
      splits = cluster_splits(tiles);
      cluster = splits > 1;
    }
  }
  const size_t k_per_split = splits > 1 ? ((k + splits - 1) / splits + bk - 1) / bk * bk : ((k + bk - 1) / bk * bk);
  if (splits > 1) splits = (unsigned)((k + k_per_split - 1) / k_per_split);
  cluster = cluster && splits > 1;

  // the tile's A and B: C's own operands, or exchanged
  const void *pa = swap ? B : A, *pb = swap ? A : B;
  const len_t la = swap ? ldb : lda, lb = swap ? lda : ldb, na = swap ? nB : nA, nb = swap ? nA : nB;
  if (swap) std::swap(a_direct, b_direct);
  CUtensorMap tmA, tmB;
  memset(&tmA, 0, sizeof(tmA));
  memset(&tmB, 0, sizeof(tmB));
  bool ok = true;
  // MN-major fp32 operands travel in the 128-byte swizzle with 32-byte atoms
  if (a_direct) {}
  else if (a_kmajor) ok = make_tmap(&tmA, bf16, pa, k, M, na, la, bk, 128, false);
  else ok = make_tmap(&tmA, bf16, pa, M, k, na, la, atom, bk, !bf16);
  if (!ok) return true;  // error recorded
  if (b_direct) {}
  else if (b_kmajor) ok = make_tmap(&tmB, bf16, pb, k, N, nb, lb, bk, persistent ? tc::kPBN / 2 : bn, false);
  else ok = make_tmap(&tmB, bf16, pb, N, k, nb, lb, atom, bk, !bf16);
  if (!ok) return true;

  tc::Params p;
  memset(&p, 0, sizeof(p));
  if (c_id == SINGLE) { p.C = static_cast<float*>(C); p.mask = static_cast<const float*>(mask); }
  else { p.Cb = static_cast<__nv_bfloat16*>(C); p.maskb = static_cast<const __nv_bfloat16*>(mask); }
  p.bias = static_cast<const float*>(bias);
  p.colsum = static_cast<float*>(colsum);
  p.c_batch_stride = (uint64_t)m * ldc;
  p.m = (uint32_t)m; p.n = (uint32_t)n; p.k = (uint32_t)k; p.ldc = (uint32_t)ldc;
  p.nA = (uint32_t)na; p.nB = (uint32_t)nb;
  p.swap = swap ? 1 : 0;
  p.a_direct = a_direct; p.b_direct = b_direct;
  if (direct) {
    p.a_src = static_cast<const float*>(pa); p.b_src = static_cast<const float*>(pb);
    p.a_ld = la; p.b_ld = lb;
    p.a_batch = (a_kmajor ? M : k) * la; p.b_batch = (b_kmajor ? N : k) * lb;
  }
  p.tiles_n = (uint32_t)((N + bn - 1) / bn);
  p.splits = splits; p.k_per_split = (uint32_t)k_per_split;
  p.alpha = (float)alpha; p.beta = (float)beta; p.epilogue = epilogue;
  p.vec_ok = c_aligned ? 1 : 0;
  p.error_flag = tc_error_flag();
  // Output through the C tensor map where the epilogue needs nothing from global memory but the bias, in the persistent kernel
  // also the mask (ZG_GEMM_TMA_EPILOGUE=0 keeps the register path)
  CUtensorMap tmC;
  memset(&tmC, 0, sizeof(tmC));
  static const bool tma_epi_on = [] { const char* e = getenv("ZG_GEMM_TMA_EPILOGUE"); return !(e && e[0] == '0'); }();
  // The unit clips a box at a whole 16-byte word: one past n would write padding columns -- a store clears them, a
  // reduction adds what the accumulator holds there (products with the repeated rows of an element-wise copied operand;
  // NaN for an infinity times a box's zero fill).  K ranges are then added element by element, which bounds the column.
  const bool tma_epi = tma_epi_on && p.vec_ok && !swap && nC <= 0x7fffffffu && n * (c_id == SINGLE ? 4 : 2) % 16 == 0;
  if (persistent) {
    const bool add = splits > 1 || (beta == 1.0 && epilogue == ZG_EPI_NONE && !colsum && c_id == SINGLE);
    CUtensorMap tmM;
    memset(&tmM, 0, sizeof(tmM));
    if (tma_epi && (add || beta == 0.0)) {
      const bool c16 = c_id == BF16;
      if (!make_tmap(&tmC, c16, C, n, m, nC, ldc, c16 ? 64 : 32, 32, false)) return true;
      if (epilogue == ZG_EPI_RELU_MASK && !make_tmap(&tmM, c16, mask, n, m, nC, ldc, c16 ? 64 : 32, 32, false)) return true;
      p.tma_epilogue = add ? (beta == 0.0 ? 3 : 2) : 1;
    }
    p.whole_tiles = (uint32_t)whole;
    const uint32_t tiles_m = (uint32_t)((m + tc::kPBM - 1) / tc::kPBM), tiles_n = (uint32_t)((n + tc::kPBN - 1) / tc::kPBN);
    const uint32_t items = (uint32_t)(whole + (ptiles - whole) * splits);
    if (p.tma_epilogue == 3)
      launch_pdl(clear_tiles_kernel, dim3(tc::kPBM / 32, (unsigned)(ptiles - whole)), dim3(256), 0, s, static_cast<float*>(C), (uint32_t)m, (uint32_t)n, (size_t)ldc,
                 (size_t)m * ldc, tiles_m, tiles_n, (uint32_t)whole);
    else if (splits > 1) prescale_c<float>(s, static_cast<float*>(C), nC, m, n, ldc, m * ldc, beta);
    if (mode == tc::kBF16) launch_persistent<tc::kBF16>(s, a_kmajor, b_kmajor, tmA, tmB, tmC, tmM, p, tiles_m, tiles_n, items);
    else launch_persistent<tc::kTF32>(s, a_kmajor, b_kmajor, tmA, tmB, tmC, tmM, p, tiles_m, tiles_n, items);
    return true;
  }
  p.cluster = cluster ? 1 : 0;
  if (splits > 1 && !cluster) prescale_c<float>(s, static_cast<float*>(C), nC, m, n, ldc, m * ldc, beta);
  dim3 grid((unsigned)((N + bn - 1) / bn * splits), (unsigned)((M + 127) / 128), (unsigned)nC);
  if (grid.y > 65535 || grid.z > 65535) return false;
  if (tma_epi && c_id == SINGLE && !cluster && !p.colsum &&
      (splits > 1 ? epilogue == ZG_EPI_NONE : (beta == 0.0 && epilogue != ZG_EPI_RELU_MASK))) {
    if (!make_tmap(&tmC, false, C, n, m, nC, ldc, 32, 32, false)) return true;
    p.tma_epilogue = splits > 1 ? 2 : 1;
  }
  if (direct) launch_tc_direct(s, bn, a_kmajor, b_kmajor, tmA, tmB, tmC, p, grid);
  else if (sums) launch_tc_mode<tc::kBF16Sums>(s, bn, a_kmajor, b_kmajor, tmA, tmB, tmC, p, grid);
  else if (mode == tc::kBF16) launch_tc_mode<tc::kBF16>(s, bn, a_kmajor, b_kmajor, tmA, tmB, tmC, p, grid);
  else if (mode == tc::kTF32) launch_tc_mode<tc::kTF32>(s, bn, a_kmajor, b_kmajor, tmA, tmB, tmC, p, grid);
  else launch_tc_mode<tc::kFP32X3>(s, bn, a_kmajor, b_kmajor, tmA, tmB, tmC, p, grid);
  return true;
}

void bmm_dispatch(dtype id, dtype c_id, cudaStream_t s, const void* A, const void* B, void* C, len_t nA, len_t nB, len_t nC, len_t m,
                  len_t n, len_t k, bool ta, bool tb, len_t lda, len_t ldb, len_t ldc, double alpha, double beta, int epilogue,
                  const void* bias, const void* mask, void* colsum) {
  g_sm_budget = g_next_sm_budget;
  g_next_sm_budget = 0;
  g_rounded = g_next_rounded;
  g_next_rounded = false;
  if (m == 0 || n == 0 || nC == 0) return;
  if (nA == 0 || nB == 0) { set_error(kBadArgument, "bmm: empty operand batch"); return; }
  if (epilogue < ZG_EPI_NONE || epilogue > ZG_EPI_RELU_MASK) { set_error(kBadArgument, "bmm: unknown epilogue %d", epilogue); return; }
  if ((epilogue == ZG_EPI_BIAS || epilogue == ZG_EPI_BIAS_RELU) && !bias) { set_error(kBadArgument, "bmm: bias epilogue without bias"); return; }
  if (epilogue == ZG_EPI_RELU_MASK && !mask) { set_error(kBadArgument, "bmm: mask epilogue without mask source"); return; }
  if (colsum && id == DOUBLE) { set_error(kUnsupported, "bmm: column sums are fp32 only"); return; }
  if (try_skinny(id, c_id, s, A, B, C, nA, nB, nC, m, n, k, ta, tb, lda, ldb, ldc, alpha, beta, epilogue, bias, mask, colsum)) return;
  if (try_tensor_core(id, c_id, s, A, B, C, nA, nB, nC, m, n, k, ta, tb, lda, ldb, ldc, alpha, beta, epilogue, bias, mask, colsum)) return;
  if (id == SINGLE && c_id == SINGLE) launch_block<float, float>(s, A, B, C, nA, nB, nC, m, n, k, ta, tb, lda, ldb, ldc, alpha, beta, epilogue, bias, mask, colsum);
  else if (id == DOUBLE && c_id == DOUBLE) launch_block<double, double>(s, A, B, C, nA, nB, nC, m, n, k, ta, tb, lda, ldb, ldc, alpha, beta, epilogue, bias, mask, colsum);
  else if (id == BF16 && c_id == SINGLE) launch_block<__nv_bfloat16, float>(s, A, B, C, nA, nB, nC, m, n, k, ta, tb, lda, ldb, ldc, alpha, beta, epilogue, bias, mask, colsum);
  else if (id == BF16 && c_id == BF16) launch_block<__nv_bfloat16, __nv_bfloat16>(s, A, B, C, nA, nB, nC, m, n, k, ta, tb, lda, ldb, ldc, alpha, beta, epilogue, bias, mask, colsum);
  else set_error(kUnsupported, "bmm: unsupported dtype combination %d -> %d", (int)id, (int)c_id);
}

// ---- the weight gradients of a network on few rows as one launch (gemm_block.cuh)
// Where the products would go to the block kernel one by one (up to 5e7 multiply-adds, see try_tensor_core), all of them
// together: above that the tensor cores gain more than the launches cost.
static bool weight_grads_ok(dtype id, const zg_weight_grad* g, len_t n, len_t rows) {
  if (id != SINGLE || n == 0 || n > (len_t)block::kGroupMax || rows == 0 || rows > 4096) return false;
  double macs = 0;
  for (len_t i = 0; i < n; ++i) {
    if (g[i].out == 0 || g[i].in == 0 || g[i].out > 0x7fffffffu || g[i].in > 0x7fffffffu || g[i].ld_dy > 0x7fffffffu || g[i].ld_x > 0x7fffffffu) return false;
    macs += (double)((g[i].out + 31) / 32 * 32) * (double)((g[i].in + 31) / 32 * 32) * (double)rows;
  }
  return macs <= 5e7;
}
extern "C" int zg_weight_grads_supported(dtype id, const zg_weight_grad* g, len_t n, len_t rows) { return weight_grads_ok(id, g, n, rows) ? 1 : 0; }

extern "C" void zg_weight_grads(dtype id, StreamWrapper w, const zg_weight_grad* g, len_t n, len_t rows, double lr) {
  if (!weight_grads_ok(id, g, n, rows)) { set_error(kUnsupported, "zg_weight_grads: dtype %d, %lu products over %lu rows", (int)id, n, rows); return; }
  block::Group q;
  memset(&q, 0, sizeof(q));
  size_t tiles = 0;
  for (len_t i = 0; i < n; ++i) {
    if (!g[i].dy || !g[i].x) { set_error(kBadArgument, "zg_weight_grads: NULL operand"); return; }
    const uint32_t tn = (uint32_t)((g[i].in + 31) / 32), tm = (uint32_t)((g[i].out + 31) / 32);
    q.item[i] = {static_cast<const float*>(g[i].dy), static_cast<const float*>(g[i].x), static_cast<float*>(g[i].dW), static_cast<float*>(g[i].W),
                 static_cast<float*>(g[i].db), static_cast<float*>(g[i].b), (uint32_t)g[i].out, (uint32_t)g[i].in, (uint32_t)g[i].ld_dy,
                 (uint32_t)g[i].ld_x, tn, (uint32_t)tiles};
    tiles += (size_t)tn * tm;
  }
  q.items = (uint32_t)n;
  q.k = (uint32_t)rows;
  q.splits = block_splits(tiles, rows);
  q.k_per_split = q.splits > 1 ? (uint32_t)(((rows + q.splits - 1) / q.splits + 7) / 8 * 8) : (uint32_t)rows;
  q.nlr = -(float)lr;  // lr cast f64 -> f32, then negated (optim.zig:103)
  using L = block::Layout<float, 32, 32, 4>;
  static SharedMemoryLimit limit;
  if (!limit.raise(block::weight_grads_kernel, L::kSmem)) return;
  launch_pdl_cluster(block::weight_grads_kernel, dim3((unsigned)(tiles * q.splits)), dim3(block::kThreads), L::kSmem, as_stream(w), q.splits, q);
}

// ---- fused middle of the MLP step (mlp_tail.cuh)
template <int CP>
static bool launch_tail_inst(cudaStream_t s, const CUtensorMap& ta, const CUtensorMap& tk, const CUtensorMap& tn, const CUtensorMap& t1,
                             const CUtensorMap& td1, const CUtensorMap& td0, const tail::Params& p, unsigned grid) {
  auto kern = tail::mlp_tail_kernel<CP>;
  static SharedMemoryLimit limit;
  if (!limit.raise(kern, tail::kSmemBytes)) return false;
  return launch_pdl(kern, dim3(grid), dim3(tail::kThreads), (size_t)tail::kSmemBytes, s, ta, tk, tn, t1, td1, td0, p);
}

template <int CP, int R, int T>
static bool launch_tail_rows(cudaStream_t s, const tail_rows::Params& p) {
  using L = tail_rows::Layout<CP, R, T>;
  auto kern = tail_rows::mlp_tail_rows_kernel<CP, R, T>;
  static SharedMemoryLimit limit;
  if (!limit.raise(kern, L::kSmem)) return false;
  return launch_pdl(kern, dim3((p.rows + R - 1) / R), dim3(T), L::kSmem, s, p);
}

void mlp_tail_launch(cudaStream_t s, len_t rows, len_t h1, len_t h2, len_t C, const void* act0, const void* W1, const void* b1, const void* W2,
                     const void* b2, const void* labels, int label_kind, len_t ld_out, double loss_div, void* act1, void* logits, void* loss_out,
                     void* dlogits, void* dact1, void* dact0, void* db2, void* db1, void* db0, int weights_ready, void* dW2) {
  if (rows == 0) return;
  if (h1 != (len_t)tail::kH1 || h2 != (len_t)tail::kH2 || C == 0 || C > (len_t)tail::kCMax) {
    set_error(kUnsupported, "zg_mlp_tail_fwd_bwd: widths %lu -> %lu -> %lu (built for %d -> %d -> at most %d)", h1, h2, C, tail::kH1, tail::kH2, tail::kCMax);
    return;
  }
  if (rows > 0x7fffffffu || ld_out < C || ld_out > 0xffffffffu) { set_error(kBadArgument, "zg_mlp_tail_fwd_bwd: rows %lu, ld_out %lu", rows, ld_out); return; }
  if (label_kind != ZG_LABEL_ONEHOT && label_kind != ZG_LABEL_INDEX) { set_error(kBadArgument, "zg_mlp_tail_fwd_bwd: unknown label kind %d", label_kind); return; }
  // no bias gradients: a grouped launch behind this one forms them with the weights' (row kernel only)
  const bool sums = db2 || db1 || db0 || rows > (len_t)sm_count() * 2 * 28;
  const void* ptrs[] = {act0, W1, b1, W2, b2, labels, act1, logits, loss_out, dlogits, dact1, dact0, sums ? db2 : act0, sums ? db1 : act0, sums ? db0 : act0};
  for (const void* q : ptrs)
    if (!q) { set_error(kBadArgument, "zg_mlp_tail_fwd_bwd: NULL argument"); return; }
  if (!host_aligned16(act0) || !host_aligned16(W1) || !host_aligned16(act1) || !host_aligned16(dact1) || !host_aligned16(dact0)) {
    set_error(kBadArgument, "zg_mlp_tail_fwd_bwd: act0, W1, act1, dact1 and dact0 must be 16-byte aligned");
    return;
  }
  if (ld_out > (len_t)tail::kCMax) { set_error(kBadArgument, "zg_mlp_tail_fwd_bwd: ld_out %lu above %d", ld_out, tail::kCMax); return; }
  const unsigned sms = (unsigned)sm_count();
  if (dW2 && rows > (len_t)sms * 2 * 28) { set_error(kUnsupported, "zg_mlp_tail_step: dW2 of %lu rows", rows); return; }
  if (rows <= (len_t)sms * 2 * 28) {  // one wave of the row kernel; 16 rows per CTA while 28 would leave SMs idle
    unsigned* counters = nullptr;
    float* partial = static_cast<float*>(workspace(s, sizeof(float) * ((rows + 15) / 16), &counters));
    if (!partial) return;
    tail_rows::Params p;
    memset(&p, 0, sizeof(p));
    p.act0 = static_cast<const float*>(act0); p.W1 = static_cast<const float*>(W1); p.W2 = static_cast<const float*>(W2);
    p.b1 = static_cast<const float*>(b1); p.b2 = static_cast<const float*>(b2);
    p.labels = labels; p.label_index = label_kind == ZG_LABEL_INDEX ? 1 : 0;
    p.act1 = static_cast<float*>(act1); p.dact1 = static_cast<float*>(dact1); p.dact0 = static_cast<float*>(dact0);
    p.logits = static_cast<float*>(logits); p.dlogits = static_cast<float*>(dlogits);
    p.db2 = static_cast<float*>(db2); p.db1 = static_cast<float*>(db1); p.db0 = static_cast<float*>(db0); p.dW2 = static_cast<float*>(dW2);
    p.loss_out = static_cast<float*>(loss_out); p.loss_partial = partial; p.counter = counters;
    p.rows = (uint32_t)rows; p.C = (uint32_t)C; p.ld_out = (uint32_t)ld_out;
    p.divisor = (float)loss_div; p.inv_divisor = 1.f / p.divisor;
    int e = 0;
    p.exact_inv = (std::frexp(p.divisor, &e) == 0.5f && std::isnormal(p.inv_divisor)) ? 1 : 0;
    p.early_weights = weights_ready ? 1 : 0;
    const bool few = rows <= (len_t)sms * 16;
#define ZG_TAIL_ROWS(CPV) few ? launch_tail_rows<CPV, 16, 256>(s, p) : launch_tail_rows<CPV, 28, 224>(s, p)
    if (C <= 4) ZG_TAIL_ROWS(4);
    else if (C <= 8) ZG_TAIL_ROWS(8);
    else if (C <= 12) ZG_TAIL_ROWS(12);
    else ZG_TAIL_ROWS(16);
#undef ZG_TAIL_ROWS
    return;
  }
  CUtensorMap tmA, tmK, tmN, tm1, tmD1, tmD0;
  // outputs leave through TMA stores of [128 rows x 32 floats] slabs (rows past the end are clipped)
  if (!make_tmap(&tm1, false, act1, tail::kH2, rows, 1, tail::kH2, 32, tail::kRows, false)) return;
  if (!make_tmap(&tmD1, false, dact1, tail::kH2, rows, 1, tail::kH2, 32, tail::kRows, false)) return;
  if (!make_tmap(&tmD0, false, dact0, tail::kH1, rows, 1, tail::kH1, 32, tail::kRows, false)) return;
  if (!make_tmap(&tmA, false, act0, tail::kH1, rows, 1, tail::kH1, 32, tail::kRows, false)) return;
  if (!make_tmap(&tmK, false, W1, tail::kH1, tail::kH2, 1, tail::kH1, 32, tail::kH2, false)) return;   // B of act0 W1^T: [n = 64 rows][k contiguous]
  if (!make_tmap(&tmN, false, W1, tail::kH1, tail::kH2, 1, tail::kH1, 32, 32, true)) return;           // B of dact1 W1: [k = 64 rows][n contiguous]
  const unsigned grid = (unsigned)((rows + tail::kRows - 1) / tail::kRows);
  unsigned* counters = nullptr;
  float* partial = static_cast<float*>(workspace(s, sizeof(float) * grid, &counters));
  if (!partial) return;
  tail::Params p;
  memset(&p, 0, sizeof(p));
  p.W2 = static_cast<const float*>(W2); p.b1 = static_cast<const float*>(b1); p.b2 = static_cast<const float*>(b2);
  p.labels = labels; p.label_index = label_kind == ZG_LABEL_INDEX ? 1 : 0;
  p.logits = static_cast<float*>(logits); p.dlogits = static_cast<float*>(dlogits);
  p.db2 = static_cast<float*>(db2); p.db1 = static_cast<float*>(db1); p.db0 = static_cast<float*>(db0);
  p.loss_out = static_cast<float*>(loss_out); p.loss_partial = partial; p.counter = counters;
  p.rows = (uint32_t)rows; p.C = (uint32_t)C; p.ld_out = (uint32_t)ld_out;
  p.divisor = (float)loss_div; p.inv_divisor = 1.f / p.divisor;
  int e = 0;
  p.exact_inv = (std::frexp(p.divisor, &e) == 0.5f && std::isnormal(p.inv_divisor)) ? 1 : 0;
  p.early_weights = weights_ready ? 1 : 0;
  p.error_flag = tc_error_flag();
  if (C <= 4) launch_tail_inst<4>(s, tmA, tmK, tmN, tm1, tmD1, tmD0, p, grid);
  else if (C <= 8) launch_tail_inst<8>(s, tmA, tmK, tmN, tm1, tmD1, tmD0, p, grid);
  else if (C <= 12) launch_tail_inst<12>(s, tmA, tmK, tmN, tm1, tmD1, tmD0, p, grid);
  else launch_tail_inst<16>(s, tmA, tmK, tmN, tm1, tmD1, tmD0, p, grid);
}

int* kernel_timeout_flag() { return tc_error_flag(); }

// Reads (and clears) the device flag that a kernel raises when one of its bounded waits runs out.
void check_tc_errors() {
  int* f = tc_error_flag();
  if (!f) return;
  int v = 0;
  if (cudaMemcpy(&v, f, sizeof(int), cudaMemcpyDeviceToHost) == cudaSuccess && v) {
    cudaDeviceSynchronize();
    cudaMemset(f, 0, sizeof(int));
    clear_workspace_tickets();  // the next launches count from zero again
    cudaDeviceSynchronize();
    set_error(kKernelTimeout, "a kernel gave up waiting on a pipeline barrier");
  }
}

// y = alpha*op(A)x + beta*y : one warp per output element of the no-trans
// case, one thread per output element (coalesced over columns) when transposed
template <typename T>
__global__ void __launch_bounds__(256) gemv_n_kernel(const T* __restrict__ A, const T* __restrict__ x, T* y, size_t m, size_t n, T alpha, T beta) {
  const int lane = threadIdx.x & 31;
  const size_t warps = ((size_t)gridDim.x * blockDim.x) >> 5;
  for (size_t r = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < m; r += warps) {
    T s = T(0);
    for (size_t j = lane; j < n; j += 32) s += A[r * n + j] * x[j];
    s = warp_sum(s);
    if (lane == 0) y[r] = (beta == T(0)) ? alpha * s : alpha * s + beta * y[r];
  }
}
template <typename T>
__global__ void __launch_bounds__(256) gemv_t_kernel(const T* __restrict__ A, const T* __restrict__ x, T* y, size_t m, size_t n, T alpha, T beta) {
  const size_t nth = (size_t)gridDim.x * blockDim.x;
  for (size_t c = (size_t)blockIdx.x * blockDim.x + threadIdx.x; c < n; c += nth) {
    T s = T(0);
    for (size_t i = 0; i < m; ++i) s += A[i * n + c] * x[i];
    y[c] = (beta == T(0)) ? alpha * s : alpha * s + beta * y[c];
  }
}
template <typename T>
__global__ void __launch_bounds__(256) ger_kernel(const T* __restrict__ a, const T* __restrict__ b, T* C, size_t m, size_t n, size_t ldc, T alpha) {
  const size_t total = m * n, nth = (size_t)gridDim.x * blockDim.x;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += nth) {
    const size_t r = i / n, c = i % n;
    C[r * ldc + c] += alpha * a[r] * b[c];
  }
}

}  // namespace zg

using namespace zg;

namespace zg {
void mlp_tail_launch(cudaStream_t s, len_t rows, len_t h1, len_t h2, len_t C, const void* act0, const void* W1, const void* b1, const void* W2,
                     const void* b2, const void* labels, int label_kind, len_t ld_out, double loss_div, void* act1, void* logits, void* loss_out,
                     void* dlogits, void* dact1, void* dact0, void* db2, void* db1, void* db0, int weights_ready, void* dW2);
}
extern "C" int zg_mlp_tail_supported(dtype id, len_t h1, len_t h2, len_t C) {
  return (id == SINGLE && g_math_mode != ZG_MATH_FFMA && h1 == (len_t)tail::kH1 && h2 == (len_t)tail::kH2 && C >= 1 && C <= (len_t)tail::kCMax) ? 1 : 0;
}
extern "C" int zg_mlp_tail_forms_dw2(len_t rows) { return rows <= (len_t)sm_count() * 2 * 28 ? 1 : 0; }
extern "C" void zg_mlp_tail_step(dtype id, StreamWrapper stream, len_t rows, len_t h1, len_t h2, len_t C, const void* act0, const void* W1,
                                 const void* b1, const void* W2, const void* b2, const void* labels, int label_kind, len_t ld_out,
                                 double loss_div, void* act1, void* logits, void* loss_out, void* dlogits, void* dact1, void* dact0,
                                 void* db2, void* db1, void* db0, int weights_ready, void* dW2) {
  if (id != SINGLE) { set_error(kUnsupported, "zg_mlp_tail_fwd_bwd: only SINGLE is implemented"); return; }
  mlp_tail_launch(as_stream(stream), rows, h1, h2, C, act0, W1, b1, W2, b2, labels, label_kind, ld_out, loss_div, act1, logits, loss_out,
                  dlogits, dact1, dact0, db2, db1, db0, weights_ready, dW2);
}
extern "C" void zg_mlp_tail_fwd_bwd(dtype id, StreamWrapper stream, len_t rows, len_t h1, len_t h2, len_t C, const void* act0, const void* W1,
                                    const void* b1, const void* W2, const void* b2, const void* labels, int label_kind, len_t ld_out,
                                    double loss_div, void* act1, void* logits, void* loss_out, void* dlogits, void* dact1, void* dact0,
                                    void* db2, void* db1, void* db0, int weights_ready) {
  if (id == SINGLE && rows > 0 && !(db2 && db1 && db0)) { set_error(kBadArgument, "zg_mlp_tail_fwd_bwd: NULL argument"); return; }
  zg_mlp_tail_step(id, stream, rows, h1, h2, C, act0, W1, b1, W2, b2, labels, label_kind, ld_out, loss_div, act1, logits, loss_out, dlogits, dact1,
                   dact0, db2, db1, db0, weights_ready, nullptr);
}

extern "C" void zg_set_math_mode(int mode) {
  if (mode < ZG_MATH_FP32X3 || mode > ZG_MATH_FFMA) { set_error(kBadArgument, "zg_set_math_mode: unknown mode %d", mode); return; }
  g_math_mode = mode;
}
extern "C" int zg_get_math_mode(void) { return g_math_mode; }

// One row of a network whose weights eight SMs read about as fast as a chain of launches starts (see mlp_forward.cuh)
constexpr size_t kFwdWeights = 200 * 1000;
extern "C" int zg_mlp_forward_supported(dtype id, len_t layers, const len_t* dims) {
  if (id != SINGLE || layers == 0 || layers > mlp_fwd::kMaxLayers) return 0;
  size_t weights = 0, inputs = 0;
  for (len_t l = 0; l < layers; ++l) {
    if (dims[l] == 0 || dims[l + 1] == 0 || dims[l] > kFwdWeights || dims[l + 1] > kFwdWeights) return 0;
    weights += dims[l] * dims[l + 1];
    inputs += (dims[l] + 3) / 4 * 4;
  }
  return weights <= kFwdWeights && inputs * sizeof(float) <= 48 * 1024;
}

extern "C" void zg_mlp_forward(dtype id, StreamWrapper w, const void* X, len_t layers, const len_t* dims, void* const* W, void* const* b,
                               void* const* out) {
  if (!zg_mlp_forward_supported(id, layers, dims)) { set_error(kUnsupported, "zg_mlp_forward: dtype %d, %lu layers", (int)id, layers); return; }
  mlp_fwd::Params p;
  memset(&p, 0, sizeof(p));
  p.X = static_cast<const float*>(X);
  p.layers = (int)layers;
  uint32_t at = 0;
  for (len_t l = 0; l < layers; ++l) {
    const uint32_t K = (uint32_t)dims[l];
    p.l[l] = {static_cast<const float*>(W[l]), static_cast<const float*>(b[l]), static_cast<float*>(out[l]), K, (uint32_t)dims[l + 1], at,
              host_aligned16(W[l]) && K % 4 == 0};
    at += (K + 3) / 4 * 4;
  }
  launch_pdl_cluster(mlp_fwd::mlp_forward_kernel, dim3(mlp_fwd::kCluster), dim3(mlp_fwd::kThreads), at * sizeof(float), as_stream(w), mlp_fwd::kCluster, p);
}

extern "C" int zg_rows_tn_supported(dtype id, len_t C) { return id == SINGLE && C >= 1 && C <= 16; }

extern "C" void zg_rows_tn(dtype id, StreamWrapper w, void* out, len_t ldo, const void* A, len_t lda, const void* x, len_t ldx, const len_t* rows,
                           len_t count, len_t N, len_t C) {
  if (!zg_rows_tn_supported(id, C)) { set_error(kUnsupported, "zg_rows_tn: dtype %d, %lu columns", (int)id, C); return; }
  if (N == 0) return;
  if (N > 0xffffffffu) { set_error(kBadArgument, "zg_rows_tn: %lu columns of A", N); return; }
  auto kern = C <= 4 ? skinny::rows_tn_kernel<4> : (C <= 8 ? skinny::rows_tn_kernel<8> : (C <= 12 ? skinny::rows_tn_kernel<12> : skinny::rows_tn_kernel<16>));
  launch_pdl(kern, dim3((unsigned)((N + 31) / 32)), dim3(skinny::kRowsThreads), 0, as_stream(w), (float*)out, (size_t)ldo, (const float*)A, (size_t)lda,
             (const float*)x, (size_t)ldx, rows, (size_t)count, (size_t)N, (int)C);
}

extern "C" void zg_bmm(dtype id, dtype c_id, StreamWrapper stream, const void* A, const void* B, void* C, len_t nA, len_t nB, len_t nC,
                       len_t m, len_t n, len_t k, bool trans_a, bool trans_b, len_t lda, len_t ldb, len_t ldc, double alpha, double beta,
                       int epilogue, const void* bias, const void* mask_src, void* colsum) {
  bmm_dispatch(id, c_id, as_stream(stream), A, B, C, nA, nB, nC, m, n, k, trans_a, trans_b, lda, ldb, ldc, alpha, beta, epilogue, bias, mask_src, colsum);
}

extern "C" void gemm(dtype id, CublasWrapper w, const void* a, const void* b, void* c, len_t m, len_t n, len_t k, bool trans_a,
                     bool trans_b, len_t lda, len_t ldb, len_t ldc, double alpha, double beta) {
  bmm_dispatch(id, id, as_stream(w), a, b, c, 1, 1, 1, m, n, k, trans_a, trans_b, lda, ldb, ldc, alpha, beta, ZG_EPI_NONE, nullptr, nullptr, nullptr);
}

extern "C" void gemv(dtype id, CublasWrapper w, const void* a, const void* x, void* y, len_t m, len_t n, bool trans_a, double alpha,
                     double beta) {
  if (m == 0 || n == 0) return;
  cudaStream_t s = as_stream(w);
  if (id == SINGLE) {
    if (trans_a) gemv_t_kernel<float><<<grid_for(n, 256), 256, 0, s>>>((const float*)a, (const float*)x, (float*)y, m, n, (float)alpha, (float)beta);
    else gemv_n_kernel<float><<<grid_for(m, 8), 256, 0, s>>>((const float*)a, (const float*)x, (float*)y, m, n, (float)alpha, (float)beta);
  } else if (id == DOUBLE) {
    if (trans_a) gemv_t_kernel<double><<<grid_for(n, 256), 256, 0, s>>>((const double*)a, (const double*)x, (double*)y, m, n, alpha, beta);
    else gemv_n_kernel<double><<<grid_for(m, 8), 256, 0, s>>>((const double*)a, (const double*)x, (double*)y, m, n, alpha, beta);
  } else { set_error(kUnsupported, "gemv: unsupported dtype %d", (int)id); return; }
  ZG_LAUNCH_CHECK();
}

extern "C" void ger(dtype id, CublasWrapper w, const void* a, const void* b, void* c, len_t m, len_t n, len_t ldc, double alpha) {
  if (m == 0 || n == 0) return;
  cudaStream_t s = as_stream(w);
  if (id == SINGLE) ger_kernel<float><<<grid_for(m * n, 1024), 256, 0, s>>>((const float*)a, (const float*)b, (float*)c, m, n, ldc, (float)alpha);
  else if (id == DOUBLE) ger_kernel<double><<<grid_for(m * n, 1024), 256, 0, s>>>((const double*)a, (const double*)b, (double*)c, m, n, ldc, alpha);
  else { set_error(kUnsupported, "ger: unsupported dtype %d", (int)id); return; }
  ZG_LAUNCH_CHECK();
}

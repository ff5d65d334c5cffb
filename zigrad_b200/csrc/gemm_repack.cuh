// Copies of operands whose rows no TMA box can address (base or row pitch no multiple of 16 bytes) with rows of whole 16-byte
// words, in a buffer of the stream's: one pass over both operands in one launch in front of a tensor-core product.
//
// For bf16 there is no other way onto the tensor cores: cp.async has no 2-byte form, and the FFMA kernel that took these
// products does 26 TFLOP/s (1000x301x501 37 us, 9.7 like this; into fp32 with sums that round, gemm_tc.cuh, 1208x1518x782 158 and 16).  For fp32 the element-wise ring (DIRECT) pays for every 4-byte copy as often as a
// slab is fetched, this once: 2047^3 134 -> 89 us.
// Bound: L1, by the reads.  A thread makes one 16-byte word of a row out of the aligned 4-byte words that hold it (five of
// them where a row of bf16 starts on an odd element); words that hold no element of the row are not read.
#pragma once

#include "common.cuh"

namespace zg {
namespace repack {

struct Operand {
  const void* src;
  void* dst;
  uint64_t ld;             // source elements per row
  uint32_t cols, words;    // elements and 16-byte words of a row
  uint64_t total;          // words of the copy
};

template <typename T>
__global__ void __launch_bounds__(256) repack_kernel(const Operand a, const Operand b) {
  constexpr int E = 16 / sizeof(T), kFlight = 2;
  pdl_sync();
  const Operand& o = blockIdx.y == 0 ? a : b;
  const uint64_t nth = (uint64_t)gridDim.x * 256;
  for (uint64_t w0 = (uint64_t)blockIdx.x * 256 + threadIdx.x; w0 < o.total; w0 += kFlight * nth) {
    uint32_t x[kFlight][5];
    bool odd[kFlight];
#pragma unroll
    for (int u = 0; u < kFlight; ++u) {
      const uint64_t w = w0 + u * nth;
#pragma unroll
      for (int j = 0; j < 5; ++j) x[u][j] = 0;
      odd[u] = false;
      if (w >= o.total) continue;
      const uint64_t row = w / o.words;
      const uint32_t c = (uint32_t)(w - row * o.words) * E, n = o.cols - c < (uint32_t)E ? o.cols - c : E;
      const uintptr_t at = reinterpret_cast<uintptr_t>(static_cast<const T*>(o.src) + row * o.ld + c);
      odd[u] = sizeof(T) == 2 && (at & 2);
      const uint32_t* p = reinterpret_cast<const uint32_t*>(at & ~(uintptr_t)3);
      const uint32_t need = (uint32_t)((at & 3) + n * sizeof(T) + 3) / 4;  // 4-byte words that hold an element
#pragma unroll
      for (int j = 0; j < 5; ++j)
        if (j < (int)need) x[u][j] = __ldg(p + j);
    }
#pragma unroll
    for (int u = 0; u < kFlight; ++u) {
      const uint64_t w = w0 + u * nth;
      if (w >= o.total) continue;
      uint4 v;
      if (odd[u]) {
        v.x = __funnelshift_r(x[u][0], x[u][1], 16); v.y = __funnelshift_r(x[u][1], x[u][2], 16);
        v.z = __funnelshift_r(x[u][2], x[u][3], 16); v.w = __funnelshift_r(x[u][3], x[u][4], 16);
      } else {
        v = make_uint4(x[u][0], x[u][1], x[u][2], x[u][3]);
      }
      // (what lies past the row's end in its last word is never read: the tensor map ends with the row)
      reinterpret_cast<uint4*>(o.dst)[w] = v;
    }
  }
}

}  // namespace repack
}  // namespace zg

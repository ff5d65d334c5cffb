// Forward pass of a small fp32 MLP on one row as one launch: act[l] = relu(W[l] act[l-1] + b[l]), none on the last.
//
// Layer by layer such a pass is a chain of launches of 3 to 4 us for a fraction of a microsecond of reading (784-128-64-10
// is 440 KB).  Here one cluster of eight CTAs walks the layers: a warp owns an output, its lanes hold the output's weights
// in registers (they do not depend on the layer before, so the first ones of the next layer are requested before the
// cluster meets), and the result goes straight into the shared memory of all eight CTAs.
// Bound by the chain (two cluster barriers and three reductions) and, as the weights grow, by what eight SMs can read.
// Measured, one row, against the chain: 784-128-64-10 5.5 us (9.1), 64-64-10 3.7 (5.0), 256-256-256-256-10 9.7 (10.9), 512-512-10 7.2
// (6.9).  More rows cost it a microsecond each and the chain nothing (784-128-64-10, 2 rows: 8.0 and 9.0; 4: 9.4 and 9.2).
#pragma once

#include <cooperative_groups.h>

#include "common.cuh"

namespace zg {
namespace mlp_fwd {

namespace cg = cooperative_groups;

constexpr int kThreads = 512, kCluster = 8, kMaxLayers = 8;
constexpr int kQuads = 8;                  // 16-byte words of a weight row per lane and chunk
constexpr uint32_t kChunk = kQuads * 128;  // floats

struct Layer {
  const float* W;  // [N, K]
  const float* b;  // [N]
  float* out;      // [N]
  uint32_t K, N, at;  // its inputs start at float `at` of shared memory
  int vec;         // W allows 16-byte reads of its rows
};
struct Params {
  const float* X;
  int layers;
  Layer l[kMaxLayers];
};

// The weights of output n from k0 on; with the first of them its bias, which would otherwise be a round trip of its own behind
// each of the cluster's barriers (784-128-64-10 5.7 -> 5.5 us, 256-256-256-256-10 10.1 -> 9.7)
__device__ __forceinline__ void fetch(float4 (&w)[kQuads], float& bias, const Layer& L, uint32_t n, uint32_t k0, int lane) {
  if (k0 == 0) bias = __ldg(L.b + n);
  const float* row = L.W + (size_t)n * L.K;
#pragma unroll
  for (int j = 0; j < kQuads; ++j) {
    const uint32_t k = k0 + (j * 32 + lane) * 4;
    w[j] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (k >= L.K) continue;
    if (L.vec) {
      w[j] = __ldg(reinterpret_cast<const float4*>(row + k));
    } else {
      w[j].x = __ldg(row + k);
      if (k + 1 < L.K) w[j].y = __ldg(row + k + 1);
      if (k + 2 < L.K) w[j].z = __ldg(row + k + 2);
      if (k + 3 < L.K) w[j].w = __ldg(row + k + 3);
    }
  }
}

static __global__ void __launch_bounds__(kThreads) mlp_forward_kernel(const __grid_constant__ Params p) {
  extern __shared__ __align__(16) float in[];
  cg::cluster_group cluster = cg::this_cluster();
  const int lane = threadIdx.x & 31;
  const uint32_t first = cluster.block_rank() * (kThreads / 32) + (threadIdx.x >> 5);
  constexpr uint32_t kStep = kCluster * (kThreads / 32);
  const Layer& last = p.l[p.layers - 1];
  for (uint32_t i = p.l[0].K + threadIdx.x; i < last.at + (last.K + 3) / 4 * 4; i += kThreads) in[i] = 0.f;  // for the words past a row's end
  pdl_sync();
  float4 w[kQuads];
  float next_bias = 0.f;
  if (first < p.l[0].N) fetch(w, next_bias, p.l[0], first, 0, lane);
  for (uint32_t i = threadIdx.x; i < p.l[0].K; i += kThreads) in[i] = p.X[i];
  cluster.sync();  // all inputs are in place, and the other CTAs run
  for (int l = 0; l < p.layers; ++l) {
    const Layer& L = p.l[l];
    const bool end = l + 1 == p.layers;
    const float* x = in + L.at;
    for (uint32_t n = first; n < L.N; n += kStep) {
      float acc = 0.f;
      const float bias = next_bias;
      for (uint32_t k0 = 0; k0 < L.K; k0 += kChunk) {
#pragma unroll
        for (int j = 0; j < kQuads; ++j) {
          const uint32_t k = k0 + (j * 32 + lane) * 4;
          if (k < L.K) {
            const float4 v = *reinterpret_cast<const float4*>(x + k);
            acc = fmaf(w[j].x, v.x, acc);
            acc = fmaf(w[j].y, v.y, acc);
            acc = fmaf(w[j].z, v.z, acc);
            acc = fmaf(w[j].w, v.w, acc);
          }
        }
        // the next weights: of this row, of this warp's next output, or of its first one in the next layer
        if (k0 + kChunk < L.K) fetch(w, next_bias, L, n, k0 + kChunk, lane);
        else if (n + kStep < L.N) fetch(w, next_bias, L, n + kStep, 0, lane);
        else if (!end && first < p.l[l + 1].N) fetch(w, next_bias, p.l[l + 1], first, 0, lane);
      }
      float v = warp_sum(acc) + bias;
      if (!end) {
        v = v > 0.f ? v : 0.f;
        if (lane < kCluster) *cluster.map_shared_rank(in + p.l[l + 1].at + n, lane) = v;
      }
      if (lane == kCluster) L.out[n] = v;
    }
    if (!end) {
      if (first >= L.N && first < p.l[l + 1].N) fetch(w, next_bias, p.l[l + 1], first, 0, lane);
      cluster.sync();
    }
  }
}

}  // namespace mlp_fwd
}  // namespace zg

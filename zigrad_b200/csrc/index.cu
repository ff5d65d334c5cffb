// Index ops: scatter_add (flat, blocked and CSR forms), CSR segment sums, row
// gather, and the GCN degree-scaled edge scatter with its backward.  Semantics:
// src/device/host_device.zig:1039-1086, :1137-1160, :1325-1351, :1356-1403 and
// src/ndarray.zig:593-633.
//
// Accumulation into shared destinations uses red.global.add.f32; the values
// added are the reference's, the order in which duplicates land is not.
#include "common.cuh"

namespace zg {

constexpr int kIThreads = 256;

template <typename T>
__global__ void __launch_bounds__(kIThreads) scatter_add_kernel(const T* __restrict__ src, const len_t* __restrict__ offs, size_t n, T* dst) {
  pdl_sync();
  const size_t nth = (size_t)gridDim.x * blockDim.x;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += nth) atomicAdd(dst + offs[i], src[i]);
}

template <typename T>
__global__ void __launch_bounds__(kIThreads) gather_rows_kernel(const T* __restrict__ src, const len_t* __restrict__ idx, size_t rows, size_t cols,
                                                                T* __restrict__ dst, len_t* __restrict__ offsets_out, int* bad) {
  pdl_sync();
  const size_t nth = (size_t)gridDim.x * blockDim.x;
  for (size_t r = (size_t)blockIdx.x * blockDim.x + threadIdx.x; r < rows; r += nth) {
    const size_t c = idx[r];
    if (c >= cols) {  // the reference returns error.IndexOutOfBounds; never read out of range
      if (bad) *bad = 1;
      dst[r] = T(0);
      if (offsets_out) offsets_out[r] = r * cols;
      continue;
    }
    const size_t o = r * cols + c;
    dst[r] = src[o];
    if (offsets_out) offsets_out[r] = o;
  }
}

// dst[tgt,:] += deg[src]*deg[tgt] * h[src,:]   -- one thread per (edge, feature)
__global__ void __launch_bounds__(kIThreads) gcn_scatter_kernel(float* dst, const float* __restrict__ h, const float* __restrict__ deg,
                                                                const len_t* __restrict__ src_idx, const len_t* __restrict__ tgt_idx,
                                                                size_t stride, size_t n_edge) {
  pdl_sync();
  const size_t total = n_edge * stride, nth = (size_t)gridDim.x * blockDim.x;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += nth) {
    const size_t e = i / stride, j = i % stride;
    const size_t s = src_idx[e], t = tgt_idx[e];
    const float w = deg[s] * deg[t];
    atomicAdd(dst + t * stride + j, w * h[s * stride + j]);
  }
}

// one thread per edge: the per-edge sums over the feature dim are formed in
// the reference's order, then added to grad_deg with one atomic each
__global__ void __launch_bounds__(kIThreads) gcn_scatter_bwd_kernel(const float* __restrict__ go, const float* __restrict__ h,
                                                                    const float* __restrict__ deg, const len_t* __restrict__ src_idx,
                                                                    const len_t* __restrict__ tgt_idx, float* grad_h, float* grad_deg,
                                                                    size_t stride, size_t n_edge) {
  pdl_sync();
  const size_t nth = (size_t)gridDim.x * blockDim.x;
  for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < n_edge; e += nth) {
    const size_t s = src_idx[e], t = tgt_idx[e];
    const float ds = deg[s], dt = deg[t];
    float gs = 0.f, gt = 0.f;
    for (size_t j = 0; j < stride; ++j) {
      const float g = go[t * stride + j];
      const float hv = h[s * stride + j];
      atomicAdd(grad_h + s * stride + j, g * ds * dt);
      gs += g * dt * hv;
      gt += g * ds * hv;
    }
    atomicAdd(grad_deg + s, gs);
    atomicAdd(grad_deg + t, gt);
  }
}

// GCN propagation over a CSR adjacency, no atomics.  A warp owns a row and FW (8, 16 or 32) features at a time.  Its lanes
// fetch index and degree scale of up to 32 neighbours at once, then 32 / FW lane groups fetch the feature rows of
// consecutive neighbours, lanes along the features: coalesced loads, all in flight together.  The products pass
// through shuffles so that every lane adds its feature up IN EDGE ORDER.
// Rows of more than kHubRow neighbours (a power-law graph of 20011 nodes has one of 1170) would be a warp's serial
// chain of round trips while everybody else is done; they are put aside and the CTA takes them together: seven warps
// fetch products into shared memory, the eighth adds the batch before in edge order, four cycles per neighbour.
// That graph, 16 features: 66 us a lane per neighbour, 32 with the loads of a warp together, 12 with hubs by CTA.
//   mode 0 = forward of scatter_gcn_deg_scaled with the edges grouped by TARGET (row = target t, col = source s):
//     out[t, j] = sum_e (deg[s] * deg[t]) * x[s, j]            (+ bias[j], ReLU)
//   mode 1 = its gradient w.r.t. h with the edges grouped by SOURCE (row = s, col = t):
//     out[s, j] = sum_e (x[t, j] * deg[s]) * deg[t]
// -- the products in the order of host_device.zig:1356-1403, the sums in edge
// order when the CSR was built by a stable sort of the edge list, which makes
// the result bit-identical to the host loops.
// Feature rows of up to NE neighbours (lane e holds node c of neighbour e).  No condition between the loads: all of them
// are in flight before the first is used (lanes past the last neighbour hold node 0, whose row is read and not added).
template <int FW, int NE>
__device__ __forceinline__ void csr_load(float (&v)[NE * FW / 32], const float* __restrict__ xj, size_t ld_x, uint32_t c, int g) {
#pragma unroll
  for (int s = 0; s < NE * FW / 32; ++s) v[s] = __ldg(xj + (size_t)__shfl_sync(0xffffffffu, c, s * (32 / FW) + g) * ld_x);
}
template <int FW, int NE>
__device__ __forceinline__ float csr_add(float acc, float (&v)[NE * FW / 32], float dc, float dr, int nk, int mode, int g, int jl) {
  constexpr int G = 32 / FW, N = NE / G;  // neighbours per step, steps
  float p[N][G];
#pragma unroll
  for (int s = 0; s < N; ++s) {
    const float de = __shfl_sync(0xffffffffu, dc, s * G + g);
    v[s] = mode == 0 ? (de * dr) * v[s] : (v[s] * dr) * de;
  }
#pragma unroll
  for (int s = 0; s < N; ++s)
#pragma unroll
    for (int e = 0; e < G; ++e) p[s][e] = __shfl_sync(0xffffffffu, v[s], e * FW + jl);
#pragma unroll
  for (int s = 0; s < N; ++s)
#pragma unroll
    for (int e = 0; e < G; ++e)
      if (s * G + e < nk) acc += p[s][e];
  return acc;
}

// VEC (many rows): rows of up to kShortRow neighbours -- most, of a graph with a handful of edges per node -- are taken FW / 4 lanes each, so
// that a warp has 4 to 16 of them in flight and a graph of 20011 nodes starts all of its chains (row bounds, neighbours, their
// features) at once instead of two or three per warp one after the other; a lane adds its four features up in edge order.
// The longer ones are dealt to the CTA's warps, a row each (a warp's own 8 or 16 rows hold up to half a dozen of them).
template <int FW>
constexpr int kShortRow = FW == 8 ? 16 : 8;  // (at 8 features 16 of them: 30000 nodes of 7.5 edges 20.5 us, with 8 21.7)
constexpr int kMiddleQueue = 512;
constexpr int kHubRow = 64, kHubQueue = 64, kGatherWarps = kIThreads / 32 - 1;

// VEC: rows of x hold whole 16-byte words at aligned addresses, and F fits into FW
template <int FW, bool VEC>
__global__ void __launch_bounds__(kIThreads) csr_gcn_propagate_kernel(float* out, const float* __restrict__ x, const float* __restrict__ deg,
                                                                      const len_t* __restrict__ row_ptr, const len_t* __restrict__ col,
                                                                      size_t n_rows, size_t F, size_t ld_x, size_t ld_out, int mode,
                                                                      int epilogue, const float* __restrict__ bias) {
  constexpr int EW = FW == 32 ? 16 : 32, kBatch = kGatherWarps * EW;  // neighbours per gathering warp, per batch
  __shared__ float batch[2][kBatch][FW];
  __shared__ uint32_t queue[kHubQueue], middle[VEC ? kMiddleQueue : 1];
  __shared__ unsigned queued, waiting;
  if (threadIdx.x == 0) queued = waiting = 0;
  __syncthreads();
  pdl_sync();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane / FW, jl = lane % FW;
  const size_t warps = ((size_t)gridDim.x * blockDim.x) >> 5, first = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  auto store = [&](size_t r, size_t j, float acc) {
    if (epilogue == ZG_EPI_BIAS || epilogue == ZG_EPI_BIAS_RELU) acc += bias[j];
    if (epilogue == ZG_EPI_BIAS_RELU) acc = acc > 0.f ? acc : 0.f;
    out[r * ld_out + j] = acc;
  };
  // a row by the whole warp, or onto the CTA's queue
  auto whole_row = [&](size_t r, len_t k0, len_t k1) {
    if (k1 - k0 > kHubRow) {
      unsigned at = 0;
      if (lane == 0) at = atomicAdd(&queued, 1u);
      at = __shfl_sync(0xffffffffu, at, 0);
      if (at < kHubQueue) {
        if (lane == 0) queue[at] = (uint32_t)r;
        return;
      }
    }
    const float dr = __ldg(deg + r);
    for (size_t j0 = 0; j0 < F; j0 += FW) {
      const bool jok = j0 + jl < F;
      const float* xj = x + j0 + (jok ? jl : 0);
      float acc = 0.f;
      for (len_t kc = k0; kc < k1; kc += 32) {
        const int nk = (int)((k1 - kc) < 32 ? (k1 - kc) : 32);
        const uint32_t c = lane < nk ? (uint32_t)__ldg(col + kc + lane) : 0u;
        const float dc = __ldg(deg + c);
        if (nk > 16) { float v[FW]; csr_load<FW, 32>(v, xj, ld_x, c, g); acc = csr_add<FW, 32>(acc, v, dc, dr, nk, mode, g, jl); }
        else if (nk > 4) { float v[FW / 2]; csr_load<FW, 16>(v, xj, ld_x, c, g); acc = csr_add<FW, 16>(acc, v, dc, dr, nk, mode, g, jl); }
        else { float v[FW / 8]; csr_load<FW, 4>(v, xj, ld_x, c, g); acc = csr_add<FW, 4>(acc, v, dc, dr, nk, mode, g, jl); }
      }
      if (jok && g == 0) store(r, j0 + jl, acc);
    }
  };
  if constexpr (VEC) {
    constexpr int LW = FW / 4, RW = 32 / LW;  // lanes per row, rows per warp
    const int sub = lane % LW;
    for (size_t r0 = first * RW; r0 < n_rows; r0 += warps * RW) {
      const size_t r = r0 + lane / LW;
      const bool in = r < n_rows;
      const len_t k0 = in ? __ldg(row_ptr + r) : 0, k1 = in ? __ldg(row_ptr + r + 1) : 0;
      const int n = k1 - k0 <= kShortRow<FW> ? (int)(k1 - k0) : 0;
      const float dr = in ? __ldg(deg + r) : 0.f;
      const size_t j = 4 * sub < F ? 4 * sub : 0;  // (lanes past the last word read the first one)
      float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int e = 0; e < kShortRow<FW>; e += 4) {
        if (!__any_sync(0xffffffffu, e < n)) break;
        uint32_t c[4];
        float d[4];
        float4 v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) c[u] = e + u < n ? (uint32_t)__ldg(col + k0 + e + u) : 0u;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          d[u] = __ldg(deg + c[u]);
          v[u] = __ldg(reinterpret_cast<const float4*>(x + (size_t)c[u] * ld_x + j));
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          if (e + u >= n) continue;
          if (mode == 0) {
            const float s = d[u] * dr;
            acc.x += s * v[u].x; acc.y += s * v[u].y; acc.z += s * v[u].z; acc.w += s * v[u].w;
          } else {
            acc.x += (v[u].x * dr) * d[u]; acc.y += (v[u].y * dr) * d[u]; acc.z += (v[u].z * dr) * d[u]; acc.w += (v[u].w * dr) * d[u];
          }
        }
      }
      if (in && k1 - k0 <= kShortRow<FW>) {
        if (4 * sub + 0 < F) store(r, 4 * sub + 0, acc.x);
        if (4 * sub + 1 < F) store(r, 4 * sub + 1, acc.y);
        if (4 * sub + 2 < F) store(r, 4 * sub + 2, acc.z);
        if (4 * sub + 3 < F) store(r, 4 * sub + 3, acc.w);
      }
      bool longer = in && sub == 0 && k1 - k0 > kShortRow<FW>;
      if (longer) {  // for whichever warp of the CTA is free
        const unsigned at = atomicAdd(&waiting, 1u);
        if (at < kMiddleQueue) {
          middle[at] = (uint32_t)r;
          longer = false;
        }
      }
      unsigned rest = __ballot_sync(0xffffffffu, longer);
      while (rest) {
        const int from = __ffs(rest) - 1;
        rest &= rest - 1;
        whole_row(r0 + from / LW, __shfl_sync(0xffffffffu, k0, from), __shfl_sync(0xffffffffu, k1, from));
      }
    }
    __syncthreads();
    const unsigned n = waiting < kMiddleQueue ? waiting : kMiddleQueue;
    for (unsigned i = warp; i < n; i += kIThreads / 32) {
      const size_t r = middle[i];
      whole_row(r, __ldg(row_ptr + r), __ldg(row_ptr + r + 1));
    }
  } else {
    for (size_t r = first; r < n_rows; r += warps) whole_row(r, __ldg(row_ptr + r), __ldg(row_ptr + r + 1));
  }
  __syncthreads();
  const unsigned hubs = queued < kHubQueue ? queued : kHubQueue;
  for (unsigned h = 0; h < hubs; ++h) {
    const size_t r = queue[h];
    const len_t k0 = __ldg(row_ptr + r), k1 = __ldg(row_ptr + r + 1);
    const float dr = __ldg(deg + r);
    for (size_t j0 = 0; j0 < F; j0 += FW) {
      const bool jok = j0 + jl < F;
      const float* xj = x + j0 + (jok ? jl : 0);
      float acc = 0.f;
      const len_t rounds = (k1 - k0 + kBatch - 1) / kBatch;
      // (the neighbours of a batch are on their way during the batch before: a gather waits for one round trip, not two)
      auto neighbour = [&](len_t kc) { return (warp > 0 && lane < EW && kc + lane < k1) ? (uint32_t)__ldg(col + kc + lane) : 0u; };
      uint32_t next = neighbour(k0 + (warp - 1) * EW);
      for (len_t i = 0; i <= rounds; ++i) {
        if (warp > 0) {
          const len_t kc = k0 + i * kBatch + (warp - 1) * EW;
          if (i < rounds && kc < k1) {
            const uint32_t c = next;
            next = neighbour(kc + kBatch);
            const float dc = __ldg(deg + c);
            constexpr int N = EW * FW / 32, G = 32 / FW;
            float v[N];
            csr_load<FW, EW>(v, xj, ld_x, c, g);
#pragma unroll
            for (int s = 0; s < N; ++s) {
              const float de = __shfl_sync(0xffffffffu, dc, s * G + g);
              batch[i & 1][(warp - 1) * EW + s * G + g][jl] = mode == 0 ? (de * dr) * v[s] : (v[s] * dr) * de;
            }
          }
        } else if (i > 0) {
          const len_t left = k1 - k0 - (i - 1) * kBatch;
          const int n = left < (len_t)kBatch ? (int)left : kBatch;
          const float* b = &batch[(i - 1) & 1][0][jl];
          int e = 0;
          for (; e + 16 <= n; e += 16) {
            float p[16];
#pragma unroll
            for (int u = 0; u < 16; ++u) p[u] = b[(e + u) * FW];
#pragma unroll
            for (int u = 0; u < 16; ++u) acc += p[u];
          }
          for (; e < n; ++e) acc += b[e * FW];
        }
        __syncthreads();
      }
      if (warp == 0 && jok && g == 0) store(r, j0 + jl, acc);
    }
  }
}

// scatter_add_2d (host_device.zig:1137-1160): dst[indices[i], :] += src[i, :] for blocks of `stride`
// contiguous elements; one thread per (block, element), consecutive threads on consecutive
// elements of a block so both sides are coalesced.
template <typename T>
__global__ void __launch_bounds__(kIThreads) scatter_add_2d_kernel(const T* __restrict__ src, const len_t* __restrict__ indices, size_t n_blocks,
                                                                   size_t stride, T* dst) {
  pdl_sync();
  const size_t total = n_blocks * stride, nth = (size_t)gridDim.x * blockDim.x;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += nth) {
    const size_t blk = i / stride, j = i - blk * stride;
    atomicAdd(dst + indices[blk] * stride + j, src[i]);
  }
}

// scatter_add_csr (host_device.zig:1325-1335): dst[j] += src[i] for j in [row_ptr[i], row_ptr[i+1]).
// A warp walks a segment; segments do not overlap, so no atomics and the result is exact.
template <typename T>
__global__ void __launch_bounds__(kIThreads) scatter_add_csr_kernel(const T* __restrict__ src, const len_t* __restrict__ row_ptr, size_t n_seg, T* dst) {
  pdl_sync();
  const int lane = threadIdx.x & 31;
  const size_t warps = ((size_t)gridDim.x * blockDim.x) >> 5;
  for (size_t r = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < n_seg; r += warps) {
    const len_t k0 = row_ptr[r], k1 = row_ptr[r + 1];
    const T v = src[r];
    for (len_t j = k0 + lane; j < k1; j += 32) dst[j] += v;
  }
}

// segment_sum_csr (host_device.zig:1337-1351): dst[i] = sum of src[row_offsets[i] .. row_offsets[i+1]).
// A warp per segment: lane l adds elements l, l+32, ... in order, then the 32 partial sums are
// folded by a shuffle tree (fixed order, so repeatable; not the host's left-to-right order).
template <typename T>
__global__ void __launch_bounds__(kIThreads) segment_sum_csr_kernel(const T* __restrict__ src, const len_t* __restrict__ row_ptr, size_t n_seg, T* __restrict__ dst) {
  pdl_sync();
  const int lane = threadIdx.x & 31;
  const size_t warps = ((size_t)gridDim.x * blockDim.x) >> 5;
  for (size_t r = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < n_seg; r += warps) {
    const len_t k0 = row_ptr[r], k1 = row_ptr[r + 1];
    T acc = T(0);
    if (k1 - k0 <= 32) {  // short segment: lane 0 adds left to right, the host's order exactly
      const T v = (k0 + lane < k1) ? src[k0 + lane] : T(0);
      for (int l = 0; l < 32; ++l) {
        const T u = __shfl_sync(0xffffffffu, v, l);
        if ((len_t)l < k1 - k0) acc += u;
      }
    } else {
      for (len_t j = k0 + lane; j < k1; j += 32) acc += src[j];
      acc = warp_sum(acc);
    }
    if (lane == 0) dst[r] = acc;
  }
}

}  // namespace zg

using namespace zg;

extern "C" void zg_scatter_add_2d(dtype id, StreamWrapper w, const void* src, const len_t* indices, len_t n_blocks, len_t stride, void* dst) {
  if (n_blocks == 0 || stride == 0) return;
  cudaStream_t s = as_stream(w);
  const unsigned g = grid_for((size_t)n_blocks * stride, kIThreads * 2);
  if (id == SINGLE) launch_pdl(scatter_add_2d_kernel<float>, dim3(g), dim3(kIThreads), 0, s, (const float*)src, indices, n_blocks, stride, (float*)dst);
  else if (id == DOUBLE) launch_pdl(scatter_add_2d_kernel<double>, dim3(g), dim3(kIThreads), 0, s, (const double*)src, indices, n_blocks, stride, (double*)dst);
  else { set_error(kUnsupported, "zg_scatter_add_2d: unsupported dtype %d", (int)id); return; }
  ZG_LAUNCH_CHECK();
}

extern "C" void zg_scatter_add_csr(dtype id, StreamWrapper w, const void* src, const len_t* row_ptr, len_t n_segments, void* dst) {
  if (n_segments == 0) return;
  cudaStream_t s = as_stream(w);
  const unsigned g = grid_for(n_segments, kIThreads / 32);
  if (id == SINGLE) launch_pdl(scatter_add_csr_kernel<float>, dim3(g), dim3(kIThreads), 0, s, (const float*)src, row_ptr, n_segments, (float*)dst);
  else if (id == DOUBLE) launch_pdl(scatter_add_csr_kernel<double>, dim3(g), dim3(kIThreads), 0, s, (const double*)src, row_ptr, n_segments, (double*)dst);
  else { set_error(kUnsupported, "zg_scatter_add_csr: unsupported dtype %d", (int)id); return; }
  ZG_LAUNCH_CHECK();
}

extern "C" void zg_segment_sum_csr(dtype id, StreamWrapper w, const void* src, const len_t* row_offsets, len_t n_segments, void* dst) {
  if (n_segments == 0) return;
  cudaStream_t s = as_stream(w);
  const unsigned g = grid_for(n_segments, kIThreads / 32);
  if (id == SINGLE) launch_pdl(segment_sum_csr_kernel<float>, dim3(g), dim3(kIThreads), 0, s, (const float*)src, row_offsets, n_segments, (float*)dst);
  else if (id == DOUBLE) launch_pdl(segment_sum_csr_kernel<double>, dim3(g), dim3(kIThreads), 0, s, (const double*)src, row_offsets, n_segments, (double*)dst);
  else { set_error(kUnsupported, "zg_segment_sum_csr: unsupported dtype %d", (int)id); return; }
  ZG_LAUNCH_CHECK();
}

extern "C" void zg_scatter_add(dtype id, StreamWrapper w, const void* src, const len_t* offsets, len_t n, void* dst) {
  if (n == 0) return;
  cudaStream_t s = as_stream(w);
  if (id == SINGLE) launch_pdl(scatter_add_kernel<float>, dim3(grid_for(n, kIThreads * 2)), dim3(kIThreads), 0, s, (const float*)src, offsets, n, (float*)dst);
  else if (id == DOUBLE) launch_pdl(scatter_add_kernel<double>, dim3(grid_for(n, kIThreads * 2)), dim3(kIThreads), 0, s, (const double*)src, offsets, n, (double*)dst);
  else { set_error(kUnsupported, "zg_scatter_add: unsupported dtype %d", (int)id); return; }
  ZG_LAUNCH_CHECK();
}

extern "C" void zg_gather_rows(dtype id, StreamWrapper w, const void* src, const len_t* idx, len_t rows, len_t cols, void* dst,
                               len_t* offsets_out) {
  if (rows == 0) return;
  cudaStream_t s = as_stream(w);
  if (id == SINGLE) launch_pdl(gather_rows_kernel<float>, dim3(grid_for(rows, kIThreads)), dim3(kIThreads), 0, s, (const float*)src, idx, rows, cols, (float*)dst, offsets_out, nullptr);
  else if (id == DOUBLE) launch_pdl(gather_rows_kernel<double>, dim3(grid_for(rows, kIThreads)), dim3(kIThreads), 0, s, (const double*)src, idx, rows, cols, (double*)dst, offsets_out, nullptr);
  else { set_error(kUnsupported, "zg_gather_rows: unsupported dtype %d", (int)id); return; }
  ZG_LAUNCH_CHECK();
}

extern "C" void zg_scatter_gcn_deg_scaled(dtype id, StreamWrapper w, void* dst, const void* h, const void* deg, const len_t* src_idx,
                                          const len_t* tgt_idx, len_t stride, len_t n_edge) {
  if (id != SINGLE) { set_error(kUnsupported, "zg_scatter_gcn_deg_scaled: only SINGLE is implemented"); return; }
  if (n_edge == 0 || stride == 0) return;
  launch_pdl(gcn_scatter_kernel, dim3(grid_for(n_edge * stride, kIThreads * 2)), dim3(kIThreads), 0, as_stream(w), (float*)dst, (const float*)h, (const float*)deg, src_idx, tgt_idx, stride, n_edge);
  ZG_LAUNCH_CHECK();
}

extern "C" void zg_scatter_gcn_deg_scaled_bwd(dtype id, StreamWrapper w, const void* grad_out, const void* h, const void* deg,
                                              const len_t* src_idx, const len_t* tgt_idx, void* grad_h, void* grad_deg, len_t stride,
                                              len_t n_edge) {
  if (id != SINGLE) { set_error(kUnsupported, "zg_scatter_gcn_deg_scaled_bwd: only SINGLE is implemented"); return; }
  if (n_edge == 0 || stride == 0) return;
  launch_pdl(gcn_scatter_bwd_kernel, dim3(grid_for(n_edge, kIThreads)), dim3(kIThreads), 0, as_stream(w), (const float*)grad_out, (const float*)h, (const float*)deg, src_idx, tgt_idx, (float*)grad_h, (float*)grad_deg, stride, n_edge);
  ZG_LAUNCH_CHECK();
}

extern "C" void zg_csr_gcn_propagate(dtype id, StreamWrapper w, void* out, const void* x, const void* deg, const len_t* row_ptr,
                                     const len_t* col_idx, len_t n_rows, len_t n_feat, len_t ld_x, len_t ld_out, int transpose_form,
                                     int epilogue, const void* bias) {
  if (id != SINGLE) { set_error(kUnsupported, "zg_csr_gcn_propagate: only SINGLE is implemented"); return; }
  if (n_rows == 0 || n_feat == 0) return;
  if (epilogue != ZG_EPI_NONE && epilogue != ZG_EPI_BIAS && epilogue != ZG_EPI_BIAS_RELU) { set_error(kBadArgument, "zg_csr_gcn_propagate: epilogue %d", epilogue); return; }
  if (epilogue != ZG_EPI_NONE && !bias) { set_error(kBadArgument, "zg_csr_gcn_propagate: bias epilogue without bias"); return; }
  if (n_rows > 0xffffffffu) { set_error(kBadArgument, "zg_csr_gcn_propagate: %lu rows", n_rows); return; }
  // lane groups as wide as the feature row: 8 features take 4 neighbours per step, 32 one
  // A warp per row while two or three waves of warps do: fewer CTAs of several rows per warp leave SMs idle, and the longer
  // rows queue up in each.  Nodes x edges per node, us, a warp per row against rows by lanes (up to 16 features / 32):
  //   500 x 7.5 3.9 and 7.5 / 4.3 and 6.7      3749 x 4.5 5.3 and 10.4 / 6.2 and 8.2     9000 x 4.5 9.2 and 8.0 / 9.4 and 9.1
  //   16000 x 7.5 12.9 and 14.6 / 16.5 and 15.3   20011 x 4.5 13.1 and 11.1 / 15.1 and 12.4   50000 x 4.5 25.8 and 16.9 / 31 and 22
  const bool vec = n_feat <= 32 && n_rows > (size_t)(n_feat <= 16 ? 128 : 64) * sm_count() && ld_x % 4 == 0 && ld_x >= (n_feat + 3) / 4 * 4 && host_aligned16(x);
  auto kern = n_feat <= 8 ? (vec ? csr_gcn_propagate_kernel<8, true> : csr_gcn_propagate_kernel<8, false>)
                          : (n_feat <= 16 ? (vec ? csr_gcn_propagate_kernel<16, true> : csr_gcn_propagate_kernel<16, false>)
                                          : (vec ? csr_gcn_propagate_kernel<32, true> : csr_gcn_propagate_kernel<32, false>));
  const size_t per_warp = vec ? (n_feat <= 8 ? 16 : (n_feat <= 16 ? 8 : 4)) : 1;
  launch_pdl(kern, dim3(grid_for(n_rows, kIThreads / 32 * per_warp)), dim3(kIThreads), 0, as_stream(w), (float*)out, (const float*)x,
             (const float*)deg, row_ptr, col_idx, (size_t)n_rows, (size_t)n_feat, (size_t)ld_x, (size_t)ld_out, transpose_form ? 1 : 0, epilogue,
             (const float*)bias);
}

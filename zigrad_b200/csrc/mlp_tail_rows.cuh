// The middle of an MLP training step (see mlp_tail.cuh for the chain of ops and its tensors) for batches whose rows fit on
// the chip at two CTAs per SM: FFMA on few rows per CTA.
//
// What bounds the kernel there is the length of the dependent chain, not its arithmetic (16 K multiply-adds per row: 8192
// rows are 2 us of the chip's FFMA rate), so the rows are spread thin: 28 per CTA (two CTAs on each of 148 SMs hold 8288
// rows), 16 while those leave SMs idle, instead of the 128 of a tensor-core tile with its operand splits and TMEM
// round trips.  The products are packed pairs (fma.rn.f32x2), which leaves every other issue slot to the shared-memory
// reads -- whose wavefronts bound the larger batches (68 % of the pipe at 8192 rows).  Measured (the op alone, replayed): 64
// rows 5.9 us, 1000 6.7, 4000 9.3, 8192 13.6, 8288 13.8; the tensor-core kernel 14.9 to 17.9 below that, 16.2 at 8289 and 16.5 at
// 16384, where this one in two waves took 28.
//
//   product 1  thread = 4 rows x 4 columns, k in pairs along 16-byte words of act0 and W1 rows (both natural layout, rows
//              132 floats apart: conflict-free); KG groups of threads share k = 128 and meet in shared memory
//   row phase  8 or 16 lanes per row, each with 8 or 4 columns of act1: partial logits, butterfly sums, then every
//              lane of a row holds all logits; the lanes share the C dlogits, each forms its columns of dact1 from all
//   product 2  thread = 4 rows x 4 consecutive columns of dact0; KG2 groups share k = 64
//   sums       bias gradients per CTA in a fixed order, one fp32 atomic per column and CTA; the loss leaves as one partial
//              per CTA with a ticket, the CTA that draws the last one folds the partials in a fixed order
//
// Weights and biases are fetched before the dependency wait when the caller vouches that the preceding kernel
// does not write them.
#pragma once

#include "common.cuh"
#include "gemm_block.cuh"

namespace zg {
namespace tail_rows {

constexpr int kH1 = 128;       // width of act0
constexpr int kH2 = 64;        // width of act1
constexpr int kCMax = 16;
constexpr int kPitch1 = kH1 + 4, kPitch2 = kH2 + 4;

struct Params {
  const float* act0;      // [rows, 128]
  const float* W1;        // [64, 128]
  const float* W2;        // [C, 64]
  const float* b1;        // [64]
  const float* b2;        // [C]
  const void* labels;     // fp32 [rows, C] one-hot / probability rows, or u64 [rows] class indices
  int label_index;
  float* act1;            // [rows, 64]
  float* logits;          // [rows, ld_out]
  float* dlogits;         // [rows, ld_out]
  float* dact1;           // [rows, 64]
  float* dact0;           // [rows, 128]
  float* db2;             // [C]   column sums are ADDED (the gradient buffer is zero at the start of a step); none: all NULL
  float* db1;             // [64]
  float* db0;             // [128]
  float* dW2;             // [C, 64] or NULL: dlogits^T act1 is ADDED, too
  float* loss_out;        // one scalar, overwritten
  float* loss_partial;    // workspace: one float per CTA
  unsigned* counter;      // workspace: ticket, zero before and after
  uint32_t rows, C, ld_out;
  float divisor, inv_divisor;
  int exact_inv;
  int early_weights;      // weights and biases may be fetched before the dependency wait
};

// the reference clamps p to [1e-7, 1 - 1e-7] before the log
constexpr float kLogPMin = -16.11809565f;     // logf(1e-7f)
constexpr float kLogPMax = -1.1920929e-07f;   // logf(1.0f - 1e-7f)

template <int CP, int R, int kThreads>
struct Layout {
  static constexpr int KG1 = kThreads / (R * kH2 / 16), KG2 = kThreads / (R * kH1 / 16);
  static constexpr int kLanes = kThreads / R, kCols = kH2 / kLanes;  // row phase: lanes per row, columns per lane
  static constexpr int kPart = R * kPitch2;
  // floats: act0 | W1 | W2 | KG1 partial tiles of product 1 (later: dact1 in the second, product 2's partial
  // tile in the third and fourth) | dlogits | labels | b1 b2 | per-warp column sums
  static constexpr int kA = 0, kW1 = kA + R * kPitch1, kW2 = kW1 + kH2 * kPitch1, kParts = kW2 + CP * kH2;
  static constexpr int kNParts = KG1 < 2 ? 2 : KG1;
  static constexpr int kDl = kParts + kNParts * kPart, kT = kDl + R * (CP + 1), kB = kT + R * CP, kSum1 = kB + kH2 + kCMax;
  static constexpr int kSum0 = kSum1 + kThreads / 32 * kH2, kFloats = kSum0 + R / 4 * kH1;
  static_assert(KG1 * R * kH2 / 16 == kThreads && KG2 * R * kH1 / 16 == kThreads && kLanes * R == kThreads && kThreads >= kH1 + kH2 + kCMax, "threads");
  static constexpr size_t kSmem = kFloats * sizeof(float);
  static_assert(KG2 == 1 || (kNParts - 2) * kPart >= R * kPitch1, "product 2's partial tile");
};

__device__ __forceinline__ void fma2(float2& d, const float2 a, const float2 b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(reinterpret_cast<uint64_t&>(d)) : "l"(reinterpret_cast<const uint64_t&>(a)), "l"(reinterpret_cast<const uint64_t&>(b)));
}
__device__ __forceinline__ void copy16(float* smem, const float* gmem, bool ok) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(smem)), "l"(gmem), "r"(ok ? 16 : 0) : "memory");
}

template <int CP, int R, int kThreads>
__global__ void __launch_bounds__(kThreads, 2) mlp_tail_rows_kernel(const Params p) {
  using L = Layout<CP, R, kThreads>;
  extern __shared__ __align__(16) float sm[];
  __shared__ float loss_warp[kThreads / 32];
  __shared__ int is_last;
  float *As = sm + L::kA, *W1s = sm + L::kW1, *W2s = sm + L::kW2, *part = sm + L::kParts, *dls = sm + L::kDl, *Ts = sm + L::kT;
  float *b1s = sm + L::kB, *b2s = b1s + kH2, *sum1 = sm + L::kSum1, *sum0 = sm + L::kSum0;
  float* dact1s = part + L::kPart;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5, C = (int)p.C;
  const uint32_t row0 = blockIdx.x * R;
  const int nrows = (int)(p.rows - row0 < (uint32_t)R ? p.rows - row0 : R);

  auto fetch_weights = [&]() {
#pragma unroll 4
    for (int e = t; e < kH2 * kH1 / 4; e += kThreads) {
      const int r = e / (kH1 / 4), c = e % (kH1 / 4) * 4;
      copy16(W1s + r * kPitch1 + c, p.W1 + r * kH1 + c, true);
    }
    for (int e = t; e < CP * kH2; e += kThreads) block::copy_async<4>(W2s + e, e < C * kH2 ? p.W2 + e : p.W2, e < C * kH2);
    if (t < kH2) block::copy_async<4>(b1s + t, p.b1 + t, true);
    else if (t < kH2 + kCMax) block::copy_async<4>(b1s + t, t < kH2 + C ? p.b2 + (t - kH2) : p.b2, t < kH2 + C);
  };
  if (p.early_weights) fetch_weights();
  pdl_sync();
  if (!p.early_weights) fetch_weights();
#pragma unroll
  for (int i = 0; i < R * kH1 / 4 / kThreads; ++i) {
    const int e = t + i * kThreads, r = e / (kH1 / 4), c = e % (kH1 / 4) * 4;
    const bool ok = r < nrows;
    copy16(As + r * kPitch1 + c, ok ? p.act0 + (size_t)(row0 + r) * kH1 + c : p.act0, ok);
  }
  if (!p.label_index) {
    const float* T = static_cast<const float*>(p.labels) + (size_t)row0 * C;
    for (int e = t; e < R * C; e += kThreads) block::copy_async<4>(Ts + e, e < nrows * C ? T + e : T, e < nrows * C);
  }
  // row phase: this thread's row and columns
  const int row = t / L::kLanes, q = t % L::kLanes;
  const bool row_ok = row < nrows;
  int lab = -1;
  if (p.label_index && row_ok) {
    const len_t l = __ldg(static_cast<const len_t*>(p.labels) + row0 + row);
    lab = l < (len_t)C ? (int)l : -1;
  }
  block::copy_commit();
  block::copy_wait<0>();
  __syncthreads();

  // ---- product 1: act0 W1^T
  {
    constexpr int kGroup = kThreads / L::KG1, kDepth = kH1 / L::KG1;
    const int g = t / kGroup, tx = t % 16, ty = t % kGroup / 16;
    const float* a = As + ty * 4 * kPitch1 + g * kDepth;
    const float* w = W1s + tx * kPitch1 + g * kDepth;
    float2 acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] = make_float2(0.f, 0.f);
#pragma unroll 4
    for (int k = 0; k < kDepth; k += 4) {
      float4 av[4], wv[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) av[i] = *reinterpret_cast<const float4*>(a + i * kPitch1 + k);
#pragma unroll
      for (int j = 0; j < 4; ++j) wv[j] = *reinterpret_cast<const float4*>(w + j * 16 * kPitch1 + k);
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          fma2(acc[i][j], make_float2(av[i].x, av[i].y), make_float2(wv[j].x, wv[j].y));
          fma2(acc[i][j], make_float2(av[i].z, av[i].w), make_float2(wv[j].z, wv[j].w));
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) part[g * L::kPart + (ty * 4 + i) * kPitch2 + tx + 16 * j] = acc[i][j].x + acc[i][j].y;
  }
  __syncthreads();

  // ---- row phase: act1, logits, loss, dlogits, dact1
  float loss = 0.f;
  {
    constexpr int NV = L::kCols / 4;  // 16-byte words per lane: columns 4 q + 32 h (8 lanes) or 4 q (16 lanes)
    float4 a1[NV];
#pragma unroll
    for (int h = 0; h < NV; ++h) {
      const int at = row * kPitch2 + 4 * q + h * 4 * L::kLanes;
      float4 v = *reinterpret_cast<const float4*>(part + at);
#pragma unroll
      for (int g = 1; g < L::KG1; ++g) {
        const float4 u = *reinterpret_cast<const float4*>(part + g * L::kPart + at);
        v.x += u.x; v.y += u.y; v.z += u.z; v.w += u.w;
      }
      const float4 b = *reinterpret_cast<const float4*>(b1s + 4 * q + h * 4 * L::kLanes);
      v.x = fmaxf(v.x + b.x, 0.f); v.y = fmaxf(v.y + b.y, 0.f); v.z = fmaxf(v.z + b.z, 0.f); v.w = fmaxf(v.w + b.w, 0.f);
      a1[h] = v;
      if (row_ok) *reinterpret_cast<float4*>(p.act1 + (size_t)(row0 + row) * kH2 + 4 * q + h * 4 * L::kLanes) = v;
    }
    float lg[CP];
#pragma unroll
    for (int c = 0; c < CP; ++c) {
      float s = 0.f;
#pragma unroll
      for (int h = 0; h < NV; ++h) {
        const float4 w = *reinterpret_cast<const float4*>(W2s + c * kH2 + 4 * q + h * 4 * L::kLanes);
        s = fmaf(a1[h].x, w.x, s); s = fmaf(a1[h].y, w.y, s); s = fmaf(a1[h].z, w.z, s); s = fmaf(a1[h].w, w.w, s);
      }
      lg[c] = s;
    }
#pragma unroll
    for (int o = 1; o < L::kLanes; o <<= 1)
#pragma unroll
      for (int c = 0; c < CP; ++c) lg[c] += __shfl_xor_sync(0xffffffffu, lg[c], o);
    float mx = -INFINITY;
#pragma unroll
    for (int c = 0; c < CP; ++c)
      if (c < C) { lg[c] += b2s[c]; mx = fmaxf(mx, lg[c]); }
    // the lanes of a row share its classes: q, q + kLanes, ..
    constexpr int NC = (CP + L::kLanes - 1) / L::kLanes;
    float own[NC], ex[NC], se = 0.f;
#pragma unroll
    for (int i = 0; i < NC; ++i) {
      own[i] = -INFINITY;
#pragma unroll
      for (int c = i * L::kLanes; c < (i + 1) * L::kLanes && c < CP; ++c)
        if (c == q + i * L::kLanes && c < C) own[i] = lg[c];
      ex[i] = __expf(own[i] - mx);  // (0 where there is no class)
      se += ex[i];
    }
#pragma unroll
    for (int o = 1; o < L::kLanes; o <<= 1) se += __shfl_xor_sync(0xffffffffu, se, o);
    const float inv = 1.f / se, lse = logf(se);
    float* gl = p.logits + (size_t)(row0 + row) * p.ld_out;
    float* gd = p.dlogits + (size_t)(row0 + row) * p.ld_out;
#pragma unroll
    for (int i = 0; i < NC; ++i) {
      const int c = q + i * L::kLanes;
      if (c < C) {
        const float tc = p.label_index ? ((c == lab) ? 1.f : 0.f) : Ts[row * C + c];
        const float diff = ex[i] * inv - tc;
        float g = 0.f;
        if (row_ok) {
          g = p.exact_inv ? diff * p.inv_divisor : diff / p.divisor;
          if (tc != 0.f) loss -= tc * fminf(fmaxf(own[i] - mx - lse, kLogPMin), kLogPMax);
          gl[c] = own[i];
          gd[c] = g;
        }
        dls[row * (CP + 1) + c] = g;
      }
    }
    __syncwarp();
    float4 x[NV];
#pragma unroll
    for (int h = 0; h < NV; ++h) x[h] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 2
    for (int c = 0; c < C; ++c) {
      const float g = dls[row * (CP + 1) + c];
#pragma unroll
      for (int h = 0; h < NV; ++h) {
        const float4 w = *reinterpret_cast<const float4*>(W2s + c * kH2 + 4 * q + h * 4 * L::kLanes);
        x[h].x = fmaf(g, w.x, x[h].x); x[h].y = fmaf(g, w.y, x[h].y); x[h].z = fmaf(g, w.z, x[h].z); x[h].w = fmaf(g, w.w, x[h].w);
      }
    }
#pragma unroll
    for (int h = 0; h < NV; ++h) {
      if (!(a1[h].x > 0.f)) x[h].x = 0.f;
      if (!(a1[h].y > 0.f)) x[h].y = 0.f;
      if (!(a1[h].z > 0.f)) x[h].z = 0.f;
      if (!(a1[h].w > 0.f)) x[h].w = 0.f;
      const int col = 4 * q + h * 4 * L::kLanes;
      if (row_ok) *reinterpret_cast<float4*>(p.dact1 + (size_t)(row0 + row) * kH2 + col) = x[h];
    }
    __syncthreads();  // the partial tiles have been read: the second one takes dact1
#pragma unroll
    for (int h = 0; h < NV; ++h) {
      const int col = 4 * q + h * 4 * L::kLanes;
      *reinterpret_cast<float4*>(dact1s + row * kPitch2 + col) = x[h];
      if (p.dW2) *reinterpret_cast<float4*>(part + row * kPitch2 + col) = a1[h];
      // column sums over the warp's rows
#pragma unroll
      for (int o = L::kLanes; o < 32; o <<= 1) {
        x[h].x += __shfl_xor_sync(0xffffffffu, x[h].x, o); x[h].y += __shfl_xor_sync(0xffffffffu, x[h].y, o);
        x[h].z += __shfl_xor_sync(0xffffffffu, x[h].z, o); x[h].w += __shfl_xor_sync(0xffffffffu, x[h].w, o);
      }
      if (lane < L::kLanes) *reinterpret_cast<float4*>(sum1 + warp * kH2 + col) = x[h];
    }
    loss = warp_sum(loss);
    if (lane == 0) loss_warp[warp] = loss;
  }
  __syncthreads();
  if (t == 0) {  // loss partial and ticket: on their way during product 2
    float s = 0.f;
#pragma unroll
    for (int w = 0; w < kThreads / 32; ++w) s += loss_warp[w];
    p.loss_partial[blockIdx.x] = s;
    __threadfence();
    is_last = atomicAdd(p.counter, 1u) == gridDim.x - 1;
    if (is_last) *p.counter = 0;
  }

  // ---- the classifier's weight gradient, whose operands are both here: a thread per class and four columns.  As a launch of
  // its own beside the other weight gradients it takes the places of the SMs that the next layer's product waits for: a step of 8192
  // rows 53.0 -> 47.2 us.
  if (p.dW2) {
    const bool wide = aligned16(p.dW2);
    for (int e = t; e < C * (kH2 / 4); e += kThreads) {
      const int c = e / (kH2 / 4), col = e % (kH2 / 4) * 4;
      float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
      for (int r = 0; r < R; ++r) {
        const float g = dls[r * (CP + 1) + c];
        const float4 a = *reinterpret_cast<const float4*>(part + r * kPitch2 + col);
        s.x = fmaf(g, a.x, s.x); s.y = fmaf(g, a.y, s.y); s.z = fmaf(g, a.z, s.z); s.w = fmaf(g, a.w, s.w);
      }
      float* dst = p.dW2 + c * kH2 + col;
      if (wide) atomicAdd(reinterpret_cast<float4*>(dst), s);
      else { atomicAdd(dst, s.x); atomicAdd(dst + 1, s.y); atomicAdd(dst + 2, s.z); atomicAdd(dst + 3, s.w); }
    }
  }

  // ---- product 2: dact1 W1, masked by act0
  {
    constexpr int kDepth = kH2 / L::KG2;
    const int g = warp / (R / 4), ty = warp % (R / 4), j = lane * 4;
    const float* d = dact1s + ty * 4 * kPitch2 + g * kDepth;
    const float* w = W1s + g * kDepth * kPitch1 + j;
    float2 acc[4][2];
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[i][0] = acc[i][1] = make_float2(0.f, 0.f);
#pragma unroll 4
    for (int k = 0; k < kDepth; k += 4) {
      float4 dv[4], wv[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) dv[i] = *reinterpret_cast<const float4*>(d + i * kPitch2 + k);
#pragma unroll
      for (int u = 0; u < 4; ++u) wv[u] = *reinterpret_cast<const float4*>(w + (k + u) * kPitch1);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float ds[4] = {dv[i].x, dv[i].y, dv[i].z, dv[i].w};
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const float2 dd = make_float2(ds[u], ds[u]);
          fma2(acc[i][0], dd, make_float2(wv[u].x, wv[u].y));
          fma2(acc[i][1], dd, make_float2(wv[u].z, wv[u].w));
        }
      }
    }
    if constexpr (L::KG2 > 1) {
      float* other = part + 2 * L::kPart;
      if (g > 0) {
#pragma unroll
        for (int i = 0; i < 4; ++i) *reinterpret_cast<float4*>(other + (ty * 4 + i) * kPitch1 + j) = make_float4(acc[i][0].x, acc[i][0].y, acc[i][1].x, acc[i][1].y);
      }
      __syncthreads();
      if (g == 0) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float4 o = *reinterpret_cast<const float4*>(other + (ty * 4 + i) * kPitch1 + j);
          acc[i][0].x += o.x; acc[i][0].y += o.y; acc[i][1].x += o.z; acc[i][1].y += o.w;
        }
      }
    }
    if (g == 0) {
      float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int r = ty * 4 + i;
        const float4 a = *reinterpret_cast<const float4*>(As + r * kPitch1 + j);
        float4 o;
        o.x = a.x > 0.f ? acc[i][0].x : 0.f; o.y = a.y > 0.f ? acc[i][0].y : 0.f;
        o.z = a.z > 0.f ? acc[i][1].x : 0.f; o.w = a.w > 0.f ? acc[i][1].y : 0.f;
        if (r < nrows) *reinterpret_cast<float4*>(p.dact0 + (size_t)(row0 + r) * kH1 + j) = o;
        s.x += o.x; s.y += o.y; s.z += o.z; s.w += o.w;
      }
      *reinterpret_cast<float4*>(sum0 + ty * kH1 + j) = s;
    }
  }
  __syncthreads();
  if (!p.db0) {
  } else if (t < kH1) {
    float s = 0.f;
#pragma unroll
    for (int w = 0; w < R / 4; ++w) s += sum0[w * kH1 + t];
    atomicAdd(p.db0 + t, s);
  } else if (t < kH1 + kH2) {
    float s = 0.f;
#pragma unroll
    for (int w = 0; w < kThreads / 32; ++w) s += sum1[w * kH2 + t - kH1];
    atomicAdd(p.db1 + t - kH1, s);
  } else if (t < kH1 + kH2 + C) {
    float s = 0.f;
#pragma unroll 8
    for (int r = 0; r < R; ++r) s += dls[r * (CP + 1) + t - kH1 - kH2];
    atomicAdd(p.db2 + t - kH1 - kH2, s);
  }
  if (is_last) {
    __threadfence();
    float v = 0.f;
    for (unsigned k = t; k < gridDim.x; k += kThreads) v += __ldcg(p.loss_partial + k);
    v = warp_sum(v);
    if (lane == 0) loss_warp[warp] = v;
    __syncthreads();
    if (t == 0) {
      float s = 0.f;
#pragma unroll
      for (int w = 0; w < kThreads / 32; ++w) s += loss_warp[w];
      *p.loss_out = s / p.divisor;
    }
  }
}

}  // namespace tail_rows
}  // namespace zg

// Multi-tensor optimizer updates over one flat parameter buffer and one flat
// gradient buffer.  Semantics: src/nn/optim.zig:100-122 (SGD), :177-234 (Adam),
// gradient clipping src/device/host_device.zig:339-346.
#include <cooperative_groups.h>

#include <cmath>
#include <cstring>

#include "common.cuh"

namespace zg {

namespace cg = cooperative_groups;

constexpr int kOThreads = 256;
constexpr int kMaxSeg = 48;  // segments per launch (table travels in kernel parameters)

struct SegTable {
  unsigned long long offset[kMaxSeg];
  unsigned long long len[kMaxSeg];
  float lr_t[kMaxSeg];  // Adam: bias-corrected step size of the segment
  // CTAs [first_cta[j], first_cta[j + 1]) work on segment j: shares that go with the lengths, so that all end together.  With
  // the same number for every segment (a second grid dimension) half of a network's CTAs were those of biases.  Norms and
  // Adam over 4 matrices of 4 to 17 M elements and their biases, behind the products of a training step (with the clock
  // those leave): 70 + 347 us, so 59 + 305; on their own, with data and clock cold, both forms take 300 to 308.
  unsigned first_cta[kMaxSeg + 1];
  int n;
  int first;  // index of the first segment of this launch in the caller's list
};

// This CTA's segment, its place among the segment's CTAs and their number
struct Share { int seg; unsigned cta, ctas; };
__device__ __forceinline__ Share share_of(const SegTable& tab) {
  int lo = 0, hi = tab.n - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (tab.first_cta[mid] <= blockIdx.x) lo = mid; else hi = mid - 1;
  }
  return {lo, blockIdx.x - tab.first_cta[lo], tab.first_cta[lo + 1] - tab.first_cta[lo]};
}

// fp32 elements from p up to the next 16-byte boundary
__device__ __forceinline__ size_t misalign_elems(const void* p) { return ((16u - (unsigned)(reinterpret_cast<uintptr_t>(p) & 15u)) & 15u) >> 2; }
__device__ __forceinline__ bool same_phase(const void* a, const void* b) {
  return ((reinterpret_cast<uintptr_t>(a) ^ reinterpret_cast<uintptr_t>(b)) & 15u) == 0;
}

// norms[first + j] = ||g_j||_2 for every segment of the table; the partial sums of its CTAs are folded by the last CTA of each segment in index order.
__global__ void __launch_bounds__(kOThreads) seg_nrm2_kernel(const float* __restrict__ g, const __grid_constant__ SegTable tab,
                                                             float* norms, double* partial, unsigned* counters, int squares) {
  __shared__ double sm[32];
  const Share sh = share_of(tab);
  const int seg = sh.seg;
  pdl_sync();
  const float* p = g + tab.offset[seg];
  const size_t n = tab.len[seg];
  const size_t nth = (size_t)sh.ctas * blockDim.x, tid = (size_t)sh.cta * blockDim.x + threadIdx.x;
  // scalar head up to the first 16-byte boundary, 128-bit body (4 loads in flight per thread), scalar tail
  size_t head = misalign_elems(p);
  if (head > n) head = n;
  float acc = 0.f, a1 = 0.f, a2 = 0.f, a3 = 0.f;
  for (size_t i = tid; i < head; i += nth) acc += p[i] * p[i];
  const float4* pv = reinterpret_cast<const float4*>(p + head);
  const size_t nv = (n - head) / 4;
  size_t v = tid;
  for (; v + 3 * nth < nv; v += 4 * nth) {
    const float4 q0 = pv[v], q1 = pv[v + nth], q2 = pv[v + 2 * nth], q3 = pv[v + 3 * nth];
    acc += q0.x * q0.x + q0.y * q0.y + q0.z * q0.z + q0.w * q0.w;
    a1 += q1.x * q1.x + q1.y * q1.y + q1.z * q1.z + q1.w * q1.w;
    a2 += q2.x * q2.x + q2.y * q2.y + q2.z * q2.z + q2.w * q2.w;
    a3 += q3.x * q3.x + q3.y * q3.y + q3.z * q3.z + q3.w * q3.w;
  }
  for (; v < nv; v += nth) {
    const float4 q0 = pv[v];
    acc += q0.x * q0.x + q0.y * q0.y + q0.z * q0.z + q0.w * q0.w;
  }
  for (size_t i = head + nv * 4 + tid; i < n; i += nth) acc += p[i] * p[i];
  acc = (acc + a1) + (a2 + a3);
  const double bs = block_sum<double>((double)acc, sm);
  double* mine = partial + tab.first_cta[seg];
  if (threadIdx.x == 0) mine[sh.cta] = bs;
  __threadfence();
  __shared__ bool last;
  if (threadIdx.x == 0) {
    const unsigned t = atomicAdd(counters + 1 + seg, 1u);
    last = (t == sh.ctas - 1);
    if (last) counters[1 + seg] = 0;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  double s = 0.0;
  for (unsigned k = threadIdx.x; k < sh.ctas; k += blockDim.x) s += __ldcg(mine + k);
  s = block_sum<double>(s, sm);
  if (threadIdx.x == 0) norms[tab.first + seg] = squares ? (float)s : (float)sqrt(s);  // squares: the caller sums them over shards first
}

__device__ __forceinline__ float clip_factor(const float* norms, int idx, float max_norm, float delta, bool* on) {
  const float nv = norms[idx];
  *on = nv > max_norm;
  return *on ? max_norm / (nv + delta) : 1.f;
}

// p += (-lr) * g, with the gradient scaled (and written back) first when its
// norm exceeds max_norm.
template <bool CLIP>
__global__ void __launch_bounds__(kOThreads) sgd_kernel(float* params, float* grads, const __grid_constant__ SegTable tab, float nlr,
                                                        const float* __restrict__ norms, float max_norm, float delta, const int zero) {
  const Share sh = share_of(tab);
  const int seg = sh.seg;
  pdl_sync();
  float* p = params + tab.offset[seg];
  float* g = grads + tab.offset[seg];
  const size_t n = tab.len[seg];
  bool on = false;
  float f = 1.f;
  if (CLIP) f = clip_factor(norms, tab.first + seg, max_norm, delta, &on);
  const size_t nth = (size_t)sh.ctas * blockDim.x;
  const size_t tid = (size_t)sh.cta * blockDim.x + threadIdx.x;
  if (same_phase(p, g) && (reinterpret_cast<uintptr_t>(p) & 3u) == 0) {
    size_t head = misalign_elems(p);
    if (head > n) head = n;
    const size_t nv = (n - head) / 4;
    for (size_t i = tid; i < head; i += nth) {
      float gi = g[i];
      if (CLIP && on) { gi *= f; g[i] = gi; }
      if (zero) g[i] = 0.f;
      p[i] = fmaf(nlr, gi, p[i]);
    }
    float4* gq = reinterpret_cast<float4*>(g + head);
    float4* pq = reinterpret_cast<float4*>(p + head);
    for (size_t v = tid; v < nv; v += nth) {
      float4 gv = gq[v];
      float4 pv = pq[v];
      if (CLIP && on) {
        gv.x *= f; gv.y *= f; gv.z *= f; gv.w *= f;
        gq[v] = gv;
      }
      if (zero) gq[v] = make_float4(0.f, 0.f, 0.f, 0.f);
      pv.x = fmaf(nlr, gv.x, pv.x); pv.y = fmaf(nlr, gv.y, pv.y); pv.z = fmaf(nlr, gv.z, pv.z); pv.w = fmaf(nlr, gv.w, pv.w);
      pq[v] = pv;
    }
    for (size_t i = head + nv * 4 + tid; i < n; i += nth) {
      float gi = g[i];
      if (CLIP && on) { gi *= f; g[i] = gi; }
      if (zero) g[i] = 0.f;
      p[i] = fmaf(nlr, gi, p[i]);
    }
  } else {
    for (size_t i = tid; i < n; i += nth) {
      float gi = g[i];
      if (CLIP && on) { gi *= f; g[i] = gi; }
      if (zero) g[i] = 0.f;
      p[i] = fmaf(nlr, gi, p[i]);
    }
  }
}

// Adam in fp32, operation for operation as the reference loop (no contraction: the file is built with --fmad=false):
//   m = b1*m + (1-b1)*g ; v = b2*v + (1-b2)*g*g ; p -= lr_t * m / (sqrt(v) + eps)
struct AdamScalars {
  float b1, b2, omb1, omb2, eps;
  __device__ __forceinline__ void apply(float g, float& m, float& v, float& p, float lr_t) const {
    m = b1 * m + omb1 * g;
    v = b2 * v + omb2 * g * g;
    p = p - lr_t * m / (sqrtf(v) + eps);
  }
  // bias-corrected step size of the tensor whose update is the t-th
  __device__ __forceinline__ float step_size(float lr, float t) const { return lr * sqrtf(1.f - powf(b2, t)) / (1.f - powf(b1, t)); }
};

// The device step counter, read before whatever this thread does next: the ticket it draws says that it has been read.
__device__ __forceinline__ unsigned long long read_counter(const unsigned long long* c) {
  unsigned long long t;
  asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(t) : "l"(c) : "memory");
  return t;
}

// `target` (or nullptr): the soft update of a target network laid out like the parameters, target = tau * p + (1 - tau) *
// target, in the same pass.
template <bool CLIP, bool BF16COPY>
__global__ void __launch_bounds__(kOThreads, 4) adam_kernel(float* params, float* grads, float* ms, float* vs, const __grid_constant__ SegTable tab,
                                                         const AdamScalars a, const float* __restrict__ norms, float max_norm,
                                                         float delta, __nv_bfloat16* copy, unsigned long long* t_dev, float lr,
                                                         unsigned* ticket, unsigned long long advance, float* target, float tau) {
  const Share sh = share_of(tab);
  const int seg = sh.seg;
  pdl_sync();
  const size_t off = tab.offset[seg];
  float* p = params + off;
  float* g = grads + off;
  float* m = ms + off;
  float* v = vs + off;
  const size_t n = tab.len[seg];
  float lr_t = tab.lr_t[seg];
  if (t_dev) {  // step counter kept on the device (graph replay): t = counter + position of this tensor
    __shared__ unsigned long long now;
    if (threadIdx.x == 0) now = read_counter(t_dev);
    __syncthreads();
    lr_t = a.step_size(lr, (float)(now + (unsigned long long)(tab.first + seg + 1)));
    // the CTA that draws the last ticket moves the counter on: by then every CTA has read it (its one reading thread draws)
    if (advance && threadIdx.x == 0 && atomicAdd(ticket, 1u) == gridDim.x - 1) {
      *ticket = 0;
      *t_dev = now + advance;
    }
  }
  bool on = false;
  float f = 1.f;
  if (CLIP) f = clip_factor(norms, tab.first + seg, max_norm, delta, &on);
  const size_t nth = (size_t)sh.ctas * blockDim.x, tid = (size_t)sh.cta * blockDim.x + threadIdx.x;
  auto one = [&](float& gi, float& mi, float& vi, float& pi) {
    if (CLIP && on) gi *= f;
    a.apply(gi, mi, vi, pi, lr_t);
  };
  auto scalar = [&](size_t i) {
    float gi = g[i], mi = m[i], vi = v[i], pi = p[i];
    one(gi, mi, vi, pi);
    if (CLIP && on) g[i] = gi;
    m[i] = mi; v[i] = vi; p[i] = pi;
    if (BF16COPY) copy[off + i] = __float2bfloat16_rn(pi);
    if (target) target[off + i] = tau * pi + (1.f - tau) * target[off + i];
  };
  size_t head = misalign_elems(p);
  if (head > n) head = n;
  bool vec = same_phase(p, g) && same_phase(p, m) && same_phase(p, v) && (reinterpret_cast<uintptr_t>(p) & 3u) == 0;
  if (target) vec = vec && same_phase(p, target + off);
  if (BF16COPY) vec = vec && (reinterpret_cast<uintptr_t>(copy + off + head) & 7u) == 0;
  if (!vec) {
    for (size_t i = tid; i < n; i += nth) scalar(i);
    return;
  }
  const size_t nv = (n - head) / 4;
  for (size_t i = tid; i < head; i += nth) scalar(i);
  float4* gq = reinterpret_cast<float4*>(g + head);
  float4* mq = reinterpret_cast<float4*>(m + head);
  float4* vq = reinterpret_cast<float4*>(v + head);
  float4* pq = reinterpret_cast<float4*>(p + head);
  auto four = [&](size_t k, float4 gv, float4 mv, float4 vv, float4 pv) {
    one(gv.x, mv.x, vv.x, pv.x);
    one(gv.y, mv.y, vv.y, pv.y);
    one(gv.z, mv.z, vv.z, pv.z);
    one(gv.w, mv.w, vv.w, pv.w);
    if (CLIP && on) gq[k] = gv;
    mq[k] = mv; vq[k] = vv; pq[k] = pv;
    if (target) {
      float4* tq = reinterpret_cast<float4*>(target + off + head) + k;
      float4 tv = *tq;
      tv.x = tau * pv.x + (1.f - tau) * tv.x; tv.y = tau * pv.y + (1.f - tau) * tv.y;
      tv.z = tau * pv.z + (1.f - tau) * tv.z; tv.w = tau * pv.w + (1.f - tau) * tv.w;
      *tq = tv;
    }
    if (BF16COPY) {
      const __nv_bfloat162 lo = __floats2bfloat162_rn(pv.x, pv.y), hi = __floats2bfloat162_rn(pv.z, pv.w);
      uint2 o;
      o.x = *reinterpret_cast<const uint32_t*>(&lo);
      o.y = *reinterpret_cast<const uint32_t*>(&hi);
      *reinterpret_cast<uint2*>(copy + off + head + 4 * k) = o;
    }
  };
  // two words of each of the four arrays in flight per thread
  size_t k = tid;
  for (; k + nth < nv; k += 2 * nth) {
    const size_t l = k + nth;
    const float4 g0 = gq[k], g1 = gq[l], m0 = mq[k], m1 = mq[l], v0 = vq[k], v1 = vq[l], p0 = pq[k], p1 = pq[l];
    four(k, g0, m0, v0, p0);
    four(l, g1, m1, v1, p1);
  }
  if (k < nv) four(k, gq[k], mq[k], vq[k], pq[k]);
  for (size_t i = head + nv * 4 + tid; i < n; i += nth) scalar(i);
}

// A step with clipping over small tensors as one launch: a cluster per tensor, whose CTAs hold its elements in registers (all
// of a thread's loads in flight at once), meet for the norm through distributed shared memory in rank order, and update.
// As two launches the update waits for the norms' kernel, its ticket and its last CTA, and reads the gradients again: 6
// tensors of up to 16 K 7.1 us, here 5.9 (SGD 5.2, 3.3).  `zero` (SGD): the applied gradients are cleared.
constexpr int kSmallThreads = 1024, kSmallItems = 4, kSmallCluster = 8;
constexpr size_t kSmallLen = (size_t)kSmallThreads * kSmallItems * kSmallCluster;
template <bool ADAM>
__global__ void __launch_bounds__(kSmallThreads) small_step_kernel(float* params, float* grads, float* ms, float* vs, const __grid_constant__ SegTable tab,
                                                                   const AdamScalars a, float* norms, float max_norm, float delta,
                                                                   unsigned long long* t_dev, float lr, unsigned* ticket,
                                                                   unsigned long long advance, float* target, float tau, int zero) {
  __shared__ double sm[32];
  __shared__ double part;
  __shared__ float step;
  cg::cluster_group cluster = cg::this_cluster();
  pdl_sync();
  const int seg = blockIdx.y;
  const size_t off = tab.offset[seg], n = tab.len[seg];
  float* p = params + off;
  float* g = grads + off;
  const size_t nth = (size_t)gridDim.x * kSmallThreads, tid = (size_t)blockIdx.x * kSmallThreads + threadIdx.x;
  float gi[kSmallItems], pi[kSmallItems], mi[kSmallItems], vi[kSmallItems], ti[kSmallItems];
#pragma unroll
  for (int i = 0; i < kSmallItems; ++i) {
    const size_t e = tid + i * nth;
    const bool ok = e < n;
    gi[i] = ok ? g[e] : 0.f;
    pi[i] = ok ? p[e] : 0.f;
    if (ADAM) {
      mi[i] = ok ? ms[off + e] : 0.f;
      vi[i] = ok ? vs[off + e] : 0.f;
      ti[i] = ok && target ? target[off + e] : 0.f;
    }
  }
  // the step size as in adam_kernel, by one thread beside the others' sums: its two powers are a chain of about a microsecond
  if (ADAM && threadIdx.x == kSmallThreads - 1) {
    step = tab.lr_t[seg];
    if (t_dev) {
      const unsigned long long t = read_counter(t_dev);
      const unsigned drawn = advance ? atomicAdd(ticket, 1u) : 0u;  // on its way while the powers are formed
      step = a.step_size(lr, (float)(t + (unsigned long long)(tab.first + seg + 1)));
      if (advance && drawn == gridDim.x * gridDim.y - 1) {
        *ticket = 0;
        *t_dev = t + advance;
      }
    }
  }
  float acc = 0.f;
#pragma unroll
  for (int i = 0; i < kSmallItems; ++i) acc += gi[i] * gi[i];
  const double bs = block_sum<double>((double)acc, sm);
  if (threadIdx.x == 0) part = bs;
  cluster.sync();
  double total = 0.0;
  for (unsigned k = 0; k < gridDim.x; ++k) total += *cluster.map_shared_rank(&part, k);
  const float norm = (float)sqrt(total), lr_t = ADAM ? step : lr;
  if (tid == 0) norms[tab.first + seg] = norm;
  const bool on = norm > max_norm;
  const float f = on ? max_norm / (norm + delta) : 1.f;
#pragma unroll
  for (int i = 0; i < kSmallItems; ++i) {
    const size_t e = tid + i * nth;
    if (e >= n) continue;
    if (on) gi[i] *= f;
    if (on || zero) g[e] = zero ? 0.f : gi[i];
    if (ADAM) {
      a.apply(gi[i], mi[i], vi[i], pi[i], lr_t);
      ms[off + e] = mi[i];
      vs[off + e] = vi[i];
      if (target) target[off + e] = tau * pi[i] + (1.f - tau) * ti[i];
    } else {
      pi[i] = fmaf(lr_t, gi[i], pi[i]);
    }
    p[e] = pi[i];
  }
  cluster.sync();  // nobody leaves while its partial sum may still be read
}

// Segments of a flat buffer set to a value: what a step clears of its gradients when the rest is about to be written.
__global__ void __launch_bounds__(kOThreads) fill_segments_kernel(float* x, const __grid_constant__ SegTable tab, float value) {
  const Share sh = share_of(tab);
  pdl_sync();
  float* p = x + tab.offset[sh.seg];
  for (size_t i = (size_t)sh.cta * blockDim.x + threadIdx.x; i < tab.len[sh.seg]; i += (size_t)sh.ctas * blockDim.x) p[i] = value;
}

__global__ void counter_add_kernel(unsigned long long* c, unsigned long long inc) {
  pdl_sync();
  *c += inc;
}

// CTAs of a tensor for small_step_kernel (an element per thread, as far as that goes: divisions and roots bound it), or 0:
// tensors too long, or more of them than run side by side
static unsigned small_cluster(const zg_segment* seg, size_t n_seg) {
  size_t mx = 0;
  for (size_t j = 0; j < n_seg; ++j) mx = seg[j].len > mx ? seg[j].len : mx;
  unsigned c = 1;
  while (c < kSmallCluster && c * (size_t)kSmallThreads < mx) c *= 2;
  return mx <= kSmallLen && n_seg <= (size_t)kMaxSeg && n_seg * c <= (size_t)sm_count() * 3 / 4 ? c : 0;
}

// Offsets, lengths and shares of the segments from `first` on: CTAs of at least four elements a thread, `per_sm` of them on an SM
static SegTable seg_table(const zg_segment* seg, size_t n_seg, size_t first, int per_sm) {
  SegTable tab;
  memset(&tab, 0, sizeof(tab));
  tab.n = (int)((n_seg - first) < (size_t)kMaxSeg ? (n_seg - first) : kMaxSeg);
  tab.first = (int)first;
  size_t total = 0;
  for (int j = 0; j < tab.n; ++j) {
    tab.offset[j] = seg[first + j].offset;
    tab.len[j] = seg[first + j].len;
    total += seg[first + j].len;
  }
  const size_t room = (size_t)sm_count() * per_sm;
  size_t per = (total + room - 1) / room, up = 0;
  if (per < (size_t)kOThreads * 4) per = (size_t)kOThreads * 4;
  for (int j = 0; j < tab.n; ++j) up += (tab.len[j] + per - 1) / per;
  // While there is room for it a segment has a CTA for its last elements as well: as a second trip of a few threads they take
  // as long again (18791 + 989 elements, Adam: 2.8 us, so 2.2).
  const bool whole = up <= room;
  for (int j = 0; j < tab.n; ++j) {
    const size_t c = (tab.len[j] + (whole ? per - 1 : per / 2)) / per;
    tab.first_cta[j + 1] = tab.first_cta[j] + (unsigned)(c < 1 ? 1 : c);
  }
  return tab;
}

static bool compute_norms(cudaStream_t s, const float* grads, const zg_segment* seg, size_t n_seg, float* norms, int squares = 0) {
  if (!norms) { set_error(kBadArgument, "optimizer: clip requested but norms scratch is NULL"); return false; }
  for (size_t first = 0; first < n_seg; first += kMaxSeg) {
    const SegTable tab = seg_table(seg, n_seg, first, 5);
    const unsigned ctas = tab.first_cta[tab.n];
    unsigned* counters = nullptr;
    double* partial = static_cast<double*>(workspace(s, sizeof(double) * ctas, &counters));
    if (!partial) return false;
    if (!launch_pdl(seg_nrm2_kernel, dim3(ctas), dim3(kOThreads), 0, s, grads, tab, norms, partial, counters, squares)) return false;
  }
  return true;
}

}  // namespace zg

using namespace zg;

extern "C" void zg_sgd_step(dtype id, StreamWrapper w, void* params, void* grads, const zg_segment* seg, len_t n_seg, double lr,
                            int clip, double max_norm, double delta, void* norms, int zero_grads) {
  if (id != SINGLE) { set_error(kUnsupported, "zg_sgd_step: only SINGLE is implemented"); return; }
  if (n_seg == 0) return;
  cudaStream_t s = as_stream(w);
  const float nlr = -(float)lr;  // lr cast f64 -> f32, then negated (optim.zig:103)
  if (const unsigned c = clip == 1 && norms ? small_cluster(seg, n_seg) : 0) {
    const SegTable tab = seg_table(seg, n_seg, 0, 1);
    launch_pdl_cluster(small_step_kernel<false>, dim3(c, (unsigned)n_seg), dim3(kSmallThreads), 0, s, c, (float*)params, (float*)grads, (float*)nullptr,
                       (float*)nullptr, tab, AdamScalars{}, (float*)norms, (float)max_norm, (float)delta, (unsigned long long*)nullptr, nlr,
                       (unsigned*)nullptr, 0ull, (float*)nullptr, 0.f, zero_grads);
    return;
  }
  if (clip == 1 && !compute_norms(s, (const float*)grads, seg, n_seg, (float*)norms)) return;
  if (clip == 2 && !norms) { set_error(kBadArgument, "optimizer: clip with given norms but norms is NULL"); return; }
  for (size_t first = 0; first < n_seg; first += kMaxSeg) {
    const SegTable tab = seg_table(seg, n_seg, first, 6);
    const dim3 grid(tab.first_cta[tab.n]);
    if (clip) launch_pdl(sgd_kernel<true>, grid, dim3(kOThreads), 0, s, (float*)params, (float*)grads, tab, nlr, (const float*)norms, (float)max_norm, (float)delta, zero_grads);
    else launch_pdl(sgd_kernel<false>, grid, dim3(kOThreads), 0, s, (float*)params, (float*)grads, tab, nlr, (const float*)nullptr, 0.f, 0.f, zero_grads);
  }
}

extern "C" void zg_fill_segments(dtype id, StreamWrapper w, void* x, const zg_segment* seg, len_t n_seg, double value) {
  if (id != SINGLE) { set_error(kUnsupported, "zg_fill_segments: only SINGLE is implemented"); return; }
  for (size_t first = 0; first < n_seg; first += kMaxSeg) {
    const SegTable tab = seg_table(seg, n_seg, first, 6);
    launch_pdl(fill_segments_kernel, dim3(tab.first_cta[tab.n]), dim3(kOThreads), 0, as_stream(w), (float*)x, tab, (float)value);
  }
}

static void adam_step(cudaStream_t s, float* P, float* G, float* M, float* V, const zg_segment* seg, len_t n_seg, len_t t_first, double lr_,
                      double beta1_, double beta2_, double eps_, int clip, double max_norm, double delta, float* norms, __nv_bfloat16* cp,
                      unsigned long long* t_dev, int advance, float* target, double tau) {
  if (n_seg == 0) return;
  const float lr = (float)lr_, beta1 = (float)beta1_, beta2 = (float)beta2_;
  const AdamScalars a{beta1, beta2, 1.f - beta1, 1.f - beta2, (float)eps_};
  if (clip && !norms) { set_error(kBadArgument, "optimizer: clip %s but norms is NULL", clip == 2 ? "with given norms" : "requested"); return; }
  auto table = [&](size_t first) {
    SegTable tab = seg_table(seg, n_seg, first, 4);
    for (int j = 0; j < tab.n; ++j) {
      const float t_f = (float)(t_first + first + j);  // counter advances once per tensor (optim.zig:189)
      tab.lr_t[j] = lr * std::sqrt(1.f - std::pow(beta2, t_f)) / (1.f - std::pow(beta1, t_f));
    }
    return tab;
  };
  // The update's last CTA moves the device counter on, by a ticket from slot 2.  On a stream whose first step is being captured
  // that slot cannot be had any more: the separate kernels then, the counter's behind them.
  const bool advances = t_dev && advance, own = advances && workspace_ready(s, 256, 2);
  unsigned* ticket = nullptr;
  if (own && !workspace(s, 256, &ticket, 2)) return;
  if (const unsigned c = clip == 1 && !cp && own == advances ? small_cluster(seg, n_seg) : 0) {
    launch_pdl_cluster(small_step_kernel<true>, dim3(c, (unsigned)n_seg), dim3(kSmallThreads), 0, s, c, P, G, M, V, table(0), a, norms, (float)max_norm,
                       (float)delta, t_dev, lr, ticket, own ? (unsigned long long)n_seg : 0ull, target, (float)tau, 0);
    return;
  }
  if (clip == 1 && !compute_norms(s, G, seg, n_seg, norms)) return;
  for (size_t first = 0; first < n_seg; first += kMaxSeg) {
    const SegTable tab = table(first);
    const dim3 grid(tab.first_cta[tab.n]), blk(kOThreads);
    const unsigned long long inc = (own && first + kMaxSeg >= n_seg) ? (unsigned long long)n_seg : 0ull;
    auto kern = clip ? (cp ? adam_kernel<true, true> : adam_kernel<true, false>) : (cp ? adam_kernel<false, true> : adam_kernel<false, false>);
    if (!launch_pdl(kern, grid, blk, 0, s, P, G, M, V, tab, a, (const float*)norms, (float)max_norm, (float)delta, cp, t_dev, lr, ticket, inc, target, (float)tau)) return;
  }
  if (advances && !own) launch_pdl(counter_add_kernel, dim3(1), dim3(1), 0, s, t_dev, (unsigned long long)n_seg);
}

extern "C" void zg_adam_step_part(dtype id, StreamWrapper w, void* params, void* grads, void* m, void* v, const zg_segment* seg, len_t n_seg,
                                  len_t t_first, double lr, double beta1, double beta2, double eps, int clip, double max_norm, double delta,
                                  void* norms, void* bf16_copy, void* step_counter, int advance_counter) {
  if (id != SINGLE) { set_error(kUnsupported, "zg_adam_step: only SINGLE is implemented"); return; }
  adam_step(as_stream(w), (float*)params, (float*)grads, (float*)m, (float*)v, seg, n_seg, t_first, lr, beta1, beta2, eps, clip, max_norm, delta,
            (float*)norms, (__nv_bfloat16*)bf16_copy, (unsigned long long*)step_counter, advance_counter, nullptr, 0.0);
}

extern "C" void zg_adam_soft_step(dtype id, StreamWrapper w, void* params, void* grads, void* m, void* v, const zg_segment* seg, len_t n_seg,
                                  len_t t_first, double lr, double beta1, double beta2, double eps, int clip, double max_norm, double delta,
                                  void* norms, void* step_counter, void* target, double tau) {
  if (id != SINGLE) { set_error(kUnsupported, "zg_adam_soft_step: only SINGLE is implemented"); return; }
  if (!target) { set_error(kBadArgument, "zg_adam_soft_step: NULL target"); return; }
  adam_step(as_stream(w), (float*)params, (float*)grads, (float*)m, (float*)v, seg, n_seg, t_first, lr, beta1, beta2, eps, clip, max_norm, delta,
            (float*)norms, nullptr, (unsigned long long*)step_counter, 1, (float*)target, tau);
}

extern "C" void zg_adam_step(dtype id, StreamWrapper w, void* params, void* grads, void* m, void* v, const zg_segment* seg, len_t n_seg,
                             len_t t_first, double lr, double beta1, double beta2, double eps, int clip, double max_norm, double delta,
                             void* norms, void* bf16_copy, void* step_counter) {
  zg_adam_step_part(id, w, params, grads, m, v, seg, n_seg, t_first, lr, beta1, beta2, eps, clip, max_norm, delta, norms, bf16_copy, step_counter, 1);
}

extern "C" void zg_segment_sumsq(dtype id, StreamWrapper w, const void* x, const zg_segment* seg, len_t n_seg, void* out) {
  if (id != SINGLE) { set_error(kUnsupported, "zg_segment_sumsq: only SINGLE is implemented"); return; }
  if (n_seg == 0) return;
  compute_norms(as_stream(w), (const float*)x, seg, n_seg, (float*)out, 1);
}

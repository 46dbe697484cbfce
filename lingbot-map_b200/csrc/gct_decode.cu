// Append-only one-token-per-frame KV cache attention ("decode" shape) for the camera head.
//
// The reference's CausalAttention (lingbot_map/layers/attention.py:90-349), as used by the camera head
// (lingbot_map/heads/camera_head.py:284-358), keeps one K and one V token per frame in a dict cache that grows by
// torch.cat every frame, is cloned, and is never evicted (the `shape[3] > 1` guard at attention.py:307); every new
// token attends to all cached tokens and to the tokens of its own call (all-true mask, attention.py:276-283).
// Here the cache is a preallocated [capacity, H, D] fp32 buffer per K and V; one kernel appends the new rows and
// computes softmax(q k^T / sqrt(D)) v for the n_q new query tokens over `cached` old + n_q new keys, fp32 throughout
// (the reference runs its heads in fp32 with autocast off).
//
// q_len is 1 (streaming) or the number of scale frames (first call), so the work is a stream over K and V:
// HBM bound, algorithmic bytes = 2 * (cached + n_q) * H * D * 4 per call.  Grid (H, splits): a CTA of eight warps owns
// one head and a contiguous range of keys.  A warp takes every eighth group of four keys and keeps two groups of K and V
// rows in flight (8 KB per warp at D = 128, 128 KB per SM with two CTAs, about three times bandwidth x latency of the HBM):
// a single row in flight per warp, as this kernel had it before, reached 1.4 TB/s.  The four dot products of a group are
// reduced together (two values change hands per step, then one), each 8-lane group exponentiates its own key, and the
// weights are broadcast.  Warps are combined through shared memory, splits through the workspace by the last CTA of each
// head to arrive (counter per head); a call of a single split writes its result directly.
#include <algorithm>

#include "gct_common.h"

namespace gct {
namespace {

constexpr int kDecodeMaxQ = 8;
constexpr int kDecodeWarps = 8;
constexpr int kAheadRows = 64;           // rows of a range sent for before the kernel before has ended: 19 MB over 288 CTAs at D = 128
constexpr int kGroup = 4;                // keys per step of a warp
constexpr float kLog2e = 1.4426950408889634f;

template <int D>
struct LaneVec;
template <>
struct LaneVec<128> {
  using T = float4;
  static __device__ __forceinline__ float dot(const T& a, const T& b) { return a.x * b.x + a.y * b.y + a.z * b.z + a.w * b.w; }
  static __device__ __forceinline__ void scale(T& acc, float f) { acc.x *= f; acc.y *= f; acc.z *= f; acc.w *= f; }
  static __device__ __forceinline__ void axpy(T& acc, float w, const T& v) {
    acc.x = fmaf(w, v.x, acc.x); acc.y = fmaf(w, v.y, acc.y); acc.z = fmaf(w, v.z, acc.z); acc.w = fmaf(w, v.w, acc.w);
  }
  static __device__ __forceinline__ T zero() { return make_float4(0.f, 0.f, 0.f, 0.f); }
};
template <>
struct LaneVec<64> {
  using T = float2;
  static __device__ __forceinline__ float dot(const T& a, const T& b) { return a.x * b.x + a.y * b.y; }
  static __device__ __forceinline__ void scale(T& acc, float f) { acc.x *= f; acc.y *= f; }
  static __device__ __forceinline__ void axpy(T& acc, float w, const T& v) { acc.x = fmaf(w, v.x, acc.x); acc.y = fmaf(w, v.y, acc.y); }
  static __device__ __forceinline__ T zero() { return make_float2(0.f, 0.f); }
};

struct DecodeArgs {
  const float* q;        // [n_q, H, D]
  const float* k_new;    // [n_q, H, D]
  const float* v_new;
  float* cache_k;        // [capacity, H, D]
  float* cache_v;
  int cached, n_q, heads, store, splits;
  float scale_log2;      // 1/sqrt(D) * log2(e): logits are base-2 exponents
  float* out;            // [n_q, H, D]
  float* part;           // [H][splits][n_q][D + 2]  (acc, m, l)
  int* counters;         // [H]
};

// kQ: 1 (streaming) or kDecodeMaxQ (any n_q up to it)
template <int D, int kQ>
__global__ void __launch_bounds__(kDecodeWarps * 32, kQ == 1 ? 2 : 1) gct_decode_attn_kernel(const DecodeArgs a) {
  using V = typename LaneVec<D>::T;
  constexpr int kPer = D / 32;
  const int h = blockIdx.x, split = blockIdx.y;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n_q = kQ == 1 ? 1 : a.n_q;
  const int total = a.cached + n_q;
  const int j0 = static_cast<int>(static_cast<long long>(split) * total / a.splits);
  const int j1 = static_cast<int>(static_cast<long long>(split + 1) * total / a.splits);
  const size_t row_stride = static_cast<size_t>(a.heads) * D;
  const size_t head_off = static_cast<size_t>(h) * D + lane * kPer;
  // Under the end of the kernel before, which leaves the memory idle: the first cached rows of the range on their way to L2.  A hint
  // that reads nothing, so it may be given for rows that kernel is still writing.  Sixteen calls at 10,000 frames 491.7 -> 477.7 us,
  // at 1,000 frames 139 -> 119; with a Linear layer of the library before each call, which lets no launch begin early, 262.7 -> 262.2.
  {
    constexpr int kLines = D * 4 / 128;
    const int rows = min(min(j1, a.cached) - j0, kAheadRows);
    for (int i = threadIdx.x; i < 2 * kLines * rows; i += kDecodeWarps * 32) {
      const float* base = i & 1 ? a.cache_v : a.cache_k;
      const int r = (i >> 1) / kLines, line = (i >> 1) % kLines;
      asm volatile("prefetch.global.L2 [%0];" ::"l"(base + static_cast<size_t>(j0 + r) * row_stride + static_cast<size_t>(h) * D + 32 * line));
    }
  }
  pdl_wait();

  // rows [j, j + kGroup) of K and V; past the end of the range the last K row again (its weight is set to zero) and zeros for
  // V, whose last row may hold an infinity
  auto load_group = [&](int j, V(&kv)[kGroup], V(&vv)[kGroup]) {
#pragma unroll
    for (int u = 0; u < kGroup; ++u) {
      const int r = min(j + u, j1 - 1);
      const float* kp = r < a.cached ? a.cache_k + static_cast<size_t>(r) * row_stride : a.k_new + static_cast<size_t>(r - a.cached) * row_stride;
      const float* vp = r < a.cached ? a.cache_v + static_cast<size_t>(r) * row_stride : a.v_new + static_cast<size_t>(r - a.cached) * row_stride;
      kv[u] = *reinterpret_cast<const V*>(kp + head_off);
      vv[u] = j + u < j1 ? *reinterpret_cast<const V*>(vp + head_off) : LaneVec<D>::zero();
    }
  };
  constexpr int kStep = kDecodeWarps * kGroup;
  V k0[kGroup], v0[kGroup], k1[kGroup], v1[kGroup];
  const int first = j0 + warp * kGroup;
  if (first < j1) load_group(first, k0, v0);

  V q[kQ], acc[kQ];
  float m[kQ], l[kQ];                      // l: this lane's share (its own key of every group)
#pragma unroll
  for (int i = 0; i < kQ; ++i) {
    q[i] = i < n_q ? *reinterpret_cast<const V*>(a.q + i * row_stride + head_off) : LaneVec<D>::zero();
    LaneVec<D>::scale(q[i], a.scale_log2);
    acc[i] = LaneVec<D>::zero();
    m[i] = -INFINITY;
    l[i] = 0.f;
  }
  // the append: the first split of each head stores the new rows (every CTA reads them from k_new / v_new)
  if (a.store && split == 0 && warp == 0) {
    for (int i = 0; i < n_q; ++i) {
      *reinterpret_cast<V*>(a.cache_k + (a.cached + i) * row_stride + head_off) = *reinterpret_cast<const V*>(a.k_new + i * row_stride + head_off);
      *reinterpret_cast<V*>(a.cache_v + (a.cached + i) * row_stride + head_off) = *reinterpret_cast<const V*>(a.v_new + i * row_stride + head_off);
    }
  }
  const int mine = lane >> 3;              // the key of a group whose logit this lane ends up with
  auto use_group = [&](int j, const V(&kv)[kGroup], const V(&vv)[kGroup]) {
    const bool valid = j + mine < j1;
#pragma unroll
    for (int i = 0; i < kQ; ++i) {
      if (kQ > 1 && i >= n_q) break;
      float d0 = LaneVec<D>::dot(q[i], kv[0]), d1 = LaneVec<D>::dot(q[i], kv[1]), d2 = LaneVec<D>::dot(q[i], kv[2]), d3 = LaneVec<D>::dot(q[i], kv[3]);
      // lanes 0-15 go on with keys 0 and 1, lanes 16-31 with 2 and 3; then one key per 8 lanes
      const bool hi = lane & 16, odd = lane & 8;
      const float e0 = (hi ? d2 : d0) + __shfl_xor_sync(0xffffffffu, hi ? d0 : d2, 16);
      const float e1 = (hi ? d3 : d1) + __shfl_xor_sync(0xffffffffu, hi ? d1 : d3, 16);
      float s = (odd ? e1 : e0) + __shfl_xor_sync(0xffffffffu, odd ? e0 : e1, 8);
      s += __shfl_xor_sync(0xffffffffu, s, 4);
      s += __shfl_xor_sync(0xffffffffu, s, 2);
      s += __shfl_xor_sync(0xffffffffu, s, 1);
      if (!valid) s = -INFINITY;
      float mn = fmaxf(s, __shfl_xor_sync(0xffffffffu, s, 8));
      mn = fmaxf(mn, __shfl_xor_sync(0xffffffffu, mn, 16));
      mn = fmaxf(mn, m[i]);                // finite: key 0 of a group is always valid
      const float alpha = exp2f(m[i] - mn), w = exp2f(s - mn);      // exp2(-inf) = 0 on the first group
      m[i] = mn;
      l[i] = fmaf(l[i], alpha, w);
      LaneVec<D>::scale(acc[i], alpha);
#pragma unroll
      for (int u = 0; u < kGroup; ++u) LaneVec<D>::axpy(acc[i], __shfl_sync(0xffffffffu, w, 8 * u), vv[u]);
    }
  };
  for (int j = first; j < j1; j += 2 * kStep) {
    if (j + kStep < j1) load_group(j + kStep, k1, v1);
    use_group(j, k0, v0);
    if (j + kStep >= j1) break;
    if (j + 2 * kStep < j1) load_group(j + 2 * kStep, k0, v0);
    use_group(j + kStep, k1, v1);
  }
  // ---- combine the warps of the CTA ----
  __shared__ float s_acc[kDecodeWarps][kQ][D];
  __shared__ float s_ml[kDecodeWarps][kQ][2];
  __shared__ int s_last;
#pragma unroll
  for (int i = 0; i < kQ; ++i) {
    if (i < n_q) {
      float ls = l[i];                     // the eight lanes of a key hold the same share
      ls += __shfl_xor_sync(0xffffffffu, ls, 8);
      ls += __shfl_xor_sync(0xffffffffu, ls, 16);
      *reinterpret_cast<V*>(&s_acc[warp][i][lane * kPer]) = acc[i];
      if (lane == 0) {
        s_ml[warp][i][0] = m[i];
        s_ml[warp][i][1] = ls;
      }
    }
  }
  __syncthreads();
  const size_t rec = D + 2;
  for (int idx = threadIdx.x; idx < n_q * D; idx += blockDim.x) {
    const int i = idx / D, d = idx - i * D;
    float mx = -INFINITY;
#pragma unroll
    for (int w = 0; w < kDecodeWarps; ++w) mx = fmaxf(mx, s_ml[w][i][0]);
    float num = 0.f, den = 0.f;
#pragma unroll
    for (int w = 0; w < kDecodeWarps; ++w) {
      const float f = exp2f(s_ml[w][i][0] - mx);      // 0 for a warp without keys
      num = fmaf(f, s_acc[w][i][d], num);
      den = fmaf(f, s_ml[w][i][1], den);
    }
    if (a.splits == 1) {
      a.out[i * row_stride + static_cast<size_t>(h) * D + d] = num / den;
    } else {
      float* p = a.part + ((static_cast<size_t>(h) * a.splits + split) * n_q + i) * rec;
      p[d] = num;
      if (d == 0) {
        p[D] = mx;
        p[D + 1] = den;
      }
    }
  }
  if (a.splits == 1) return;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    const int prev = atomicAdd(a.counters + h, 1);
    s_last = prev == a.splits - 1;
    if (s_last) a.counters[h] = 0;
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  // ---- last CTA of this head: merge the splits ----
  for (int idx = threadIdx.x; idx < n_q * D; idx += blockDim.x) {
    const int i = idx / D, d = idx - i * D;
    const float* p0 = a.part + (static_cast<size_t>(h) * a.splits * n_q + i) * rec;
    const size_t step = n_q * rec;
    float mx = -INFINITY;
#pragma unroll 8
    for (int s = 0; s < a.splits; ++s) mx = fmaxf(mx, __ldcg(p0 + s * step + D));
    float num = 0.f, den = 0.f;
#pragma unroll 8
    for (int s = 0; s < a.splits; ++s) {
      const float* p = p0 + s * step;
      const float f = exp2f(__ldcg(p + D) - mx);
      num = fmaf(f, __ldcg(p + d), num);
      den = fmaf(f, __ldcg(p + D + 1), den);
    }
    a.out[i * row_stride + static_cast<size_t>(h) * D + d] = num / den;
  }
}

}  // namespace

size_t decode_counter_bytes(int heads) { return (static_cast<size_t>(heads) * sizeof(int) + 255) & ~size_t(255); }
size_t decode_workspace_bytes(int heads, int head_dim, int splits, int n_q) {
  return decode_counter_bytes(heads) + static_cast<size_t>(heads) * splits * n_q * (head_dim + 2) * sizeof(float);
}

int launch_decode_attention(const float* q, const float* k_new, const float* v_new, int n_q, float* cache_k, float* cache_v,
                            int cached, int capacity, int store, int heads, int head_dim, float* out, void* workspace,
                            size_t workspace_bytes, cudaStream_t stream) {
  if (q == nullptr || k_new == nullptr || v_new == nullptr || cache_k == nullptr || cache_v == nullptr || out == nullptr ||
      workspace == nullptr)
    return fail(GCT_ERR_INVALID, "decode attention: null argument");
  if (head_dim != 64 && head_dim != 128) return fail(GCT_ERR_INVALID, "decode attention: head_dim must be 64 or 128");
  if (n_q < 1 || n_q > kDecodeMaxQ) return fail(GCT_ERR_INVALID, "decode attention: 1..8 new tokens per call");
  if (heads < 1 || cached < 0 || capacity < cached + (store ? n_q : 0))
    return fail(GCT_ERR_CAPACITY, "decode attention: cache capacity of " + std::to_string(capacity) + " rows exceeded");
  auto misaligned = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) != 0; };
  if (misaligned(q) || misaligned(k_new) || misaligned(v_new) || misaligned(cache_k) || misaligned(cache_v) || misaligned(out) ||
      (reinterpret_cast<uintptr_t>(workspace) & 255) != 0)
    return fail(GCT_ERR_INVALID, "decode attention: tensors must be 16-byte aligned, the workspace 256-byte aligned");
  int sms = 148;
  const int rc = device_sm_count(&sms);
  if (rc != GCT_OK) return rc;
  const int total = cached + n_q;
  // Two CTAs per SM, at least 64 keys each (two steps of the eight warps: below that the merge costs more): one wave for a single
  // new token; for two to eight at D = 128 a CTA fills the registers of an SM (190 per thread) and they are two waves.
  int splits = std::max(1, std::min(2 * sms / heads, (total + 63) / 64));
  while (splits > 1 && decode_workspace_bytes(heads, head_dim, splits, n_q) > workspace_bytes) --splits;
  if (decode_workspace_bytes(heads, head_dim, splits, n_q) > workspace_bytes)
    return fail(GCT_ERR_CAPACITY, "decode attention: workspace too small");
  DecodeArgs a;
  a.q = q;
  a.k_new = k_new;
  a.v_new = v_new;
  a.cache_k = cache_k;
  a.cache_v = cache_v;
  a.cached = cached;
  a.n_q = n_q;
  a.heads = heads;
  a.store = store;
  a.splits = splits;
  a.scale_log2 = kLog2e / sqrtf(static_cast<float>(head_dim));
  a.out = out;
  a.counters = static_cast<int*>(workspace);                       // zeroed by the caller once; the kernel rezeroes
  a.part = reinterpret_cast<float*>(static_cast<uint8_t*>(workspace) + decode_counter_bytes(heads));
  const dim3 grid(heads, splits);
  const dim3 block(kDecodeWarps * 32);
  auto kernel = head_dim == 128 ? (n_q == 1 ? gct_decode_attn_kernel<128, 1> : gct_decode_attn_kernel<128, kDecodeMaxQ>)
                                : (n_q == 1 ? gct_decode_attn_kernel<64, 1> : gct_decode_attn_kernel<64, kDecodeMaxQ>);
  GCT_CUDA_CHECK(launch_pdl(kernel, grid, block, 0, stream, a));
  return GCT_OK;
}

}  // namespace gct

extern "C" {

int gct_decode_workspace_bytes(int heads, int head_dim, size_t* bytes_out) {
  if (heads < 1 || (head_dim != 64 && head_dim != 128) || bytes_out == nullptr)
    return gct::fail(GCT_ERR_INVALID, "gct_decode_workspace_bytes: bad argument");
  *bytes_out = gct::decode_workspace_bytes(heads, head_dim, 32, gct::kDecodeMaxQ);
  return GCT_OK;
}

int gct_decode_attention(const float* q_dev, const float* k_new_dev, const float* v_new_dev, int n_new, float* cache_k_dev,
                         float* cache_v_dev, int cached, int capacity, int store, int heads, int head_dim, float* out_dev,
                         void* workspace_dev, size_t workspace_bytes, void* stream) {
  return gct::launch_decode_attention(q_dev, k_new_dev, v_new_dev, n_new, cache_k_dev, cache_v_dev, cached, capacity, store,
                                      heads, head_dim, out_dev, workspace_dev, workspace_bytes, static_cast<cudaStream_t>(stream));
}

}  // extern "C"

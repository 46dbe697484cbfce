// HBM-bound helpers around the attention kernel: fused q/k LayerNorm + RoPE + bf16 cast with the
// K/V rows written straight into their cache pages, fp32->bf16 cast, split-KV merge, RoPE tables.
#include <math.h>

#include <type_traits>

#include "gct_common.h"

namespace gct {
namespace {

struct Row8 {
  float v[8];
};

__device__ __forceinline__ Row8 load8(const void* base, int dtype, size_t elem) {
  Row8 r;
  if (dtype == GCT_F32) {
    const float4 a = *reinterpret_cast<const float4*>(static_cast<const float*>(base) + elem);
    const float4 b = *reinterpret_cast<const float4*>(static_cast<const float*>(base) + elem + 4);
    r.v[0] = a.x; r.v[1] = a.y; r.v[2] = a.z; r.v[3] = a.w;
    r.v[4] = b.x; r.v[5] = b.y; r.v[6] = b.z; r.v[7] = b.w;
  } else {
    const uint4 u = *reinterpret_cast<const uint4*>(static_cast<const __nv_bfloat16*>(base) + elem);
    const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w[i]));
      r.v[2 * i] = f.x;
      r.v[2 * i + 1] = f.y;
    }
  }
  return r;
}

__device__ __forceinline__ void store8(__nv_bfloat16* dst, const Row8& r) {
  uint4 u;
  __nv_bfloat162 p0 = __floats2bfloat162_rn(r.v[0], r.v[1]), p1 = __floats2bfloat162_rn(r.v[2], r.v[3]);
  __nv_bfloat162 p2 = __floats2bfloat162_rn(r.v[4], r.v[5]), p3 = __floats2bfloat162_rn(r.v[6], r.v[7]);
  u.x = *reinterpret_cast<uint32_t*>(&p0);
  u.y = *reinterpret_cast<uint32_t*>(&p1);
  u.z = *reinterpret_cast<uint32_t*>(&p2);
  u.w = *reinterpret_cast<uint32_t*>(&p3);
  *reinterpret_cast<uint4*>(dst) = u;
}

// sum over the eight lanes of a row
__device__ __forceinline__ float row_sum(float x) {
  x += __shfl_xor_sync(0xffffffffu, x, 1);
  x += __shfl_xor_sync(0xffffffffu, x, 2);
  x += __shfl_xor_sync(0xffffffffu, x, 4);
  return x;
}

// ---- q/k LayerNorm + RoPE + bf16 + page write ------------------------------------------------------
//   LayerNorm(64), eps 1e-5, affine            lingbot_map/layers/attention.py:58-59,415
//   3-D RoPE: pair (2m,2m+1) rotated by angle m lingbot_map/layers/rope.py:450-461
//   2-D RoPE: inside each 32-wide half pair (j, j+16) rotated by angle j; table entry 16*half + j
//                                              lingbot_map/layers/rope.py:134-157,191-198
//   page write of K/V rows                     lingbot_map/layers/flashinfer_cache.py:503-505,547-549
//
// Four lanes per (token, head) row of 64, rows handed to the lanes in order (any number of heads fills the warps).  Lane part s
// owns elements [e, e+8) and [e+16, e+24) with e = 32*(s/2) + 8*(s%2): the partners of both rotations are then its own, the
// only exchanges are the two steps of each LayerNorm sum, and q, k and v are six 16-byte loads in flight (twelve in fp32).
// With one frame (12 MB, 1005 rows of 16 heads) the kernel is one round trip to memory and its launch; with many it is bound by
// memory and by instructions.  What it is built around: types and rotation are template parameters, because a branch on the
// type at each load makes the loads wait for one another; norm parameters are read once per CTA into shared memory under the
// row loads.  With eight lanes per row and types at
// run time (31 shuffles per four heads instead of 10 per eight, three round trips in a row) one frame took 8.5 us (2-D) and 9.9 us (3-D,
// pages), now 6.0 and 6.4 us; eight frames (99 MB) 31.5 us, now 21.2 us (4.7 TB/s).
constexpr int kPrepThreads = 128;
constexpr int kRope3dF64 = 3;            // GCT_ROPE_3D on a table of doubles

template <bool kF32>
struct RawRow;                           // a lane's sixteen elements as loaded
template <>
struct RawRow<false> {
  uint4 u[2];
  __device__ __forceinline__ void load(const void* base, size_t e) {
    const __nv_bfloat16* p = static_cast<const __nv_bfloat16*>(base) + e;
    u[0] = *reinterpret_cast<const uint4*>(p);
    u[1] = *reinterpret_cast<const uint4*>(p + 16);
  }
  __device__ __forceinline__ void floats(float (&x)[16]) const {
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const uint32_t w[4] = {u[c].x, u[c].y, u[c].z, u[c].w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w[i]));
        x[8 * c + 2 * i] = f.x;
        x[8 * c + 2 * i + 1] = f.y;
      }
    }
  }
};
template <>
struct RawRow<true> {
  float4 u[4];
  __device__ __forceinline__ void load(const void* base, size_t e) {
    const float4* p = reinterpret_cast<const float4*>(static_cast<const float*>(base) + e);
    u[0] = p[0];
    u[1] = p[1];
    u[2] = p[4];
    u[3] = p[5];
  }
  __device__ __forceinline__ void floats(float (&x)[16]) const {
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      x[4 * c] = u[c].x;
      x[4 * c + 1] = u[c].y;
      x[4 * c + 2] = u[c].z;
      x[4 * c + 3] = u[c].w;
    }
  }
};

__device__ __forceinline__ void store16(__nv_bfloat16* dst, const float (&x)[16]) {
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    Row8 r;
#pragma unroll
    for (int i = 0; i < 8; ++i) r.v[i] = x[8 * c + i];
    store8(dst + 16 * c, r);
  }
}

// sum over the four lanes of a row
__device__ __forceinline__ float quad_sum(float x) {
  x += __shfl_xor_sync(0xffffffffu, x, 1);
  x += __shfl_xor_sync(0xffffffffu, x, 2);
  return x;
}

// w, bia: 64 floats each in shared memory, already offset by the lane's first element.
__device__ __forceinline__ void norm16(float (&x)[16], const float* w, const float* bia) {
  float s[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int i = 0; i < 16; ++i) s[i & 3] += x[i];
  const float mean = quad_sum((s[0] + s[1]) + (s[2] + s[3])) * (1.f / 64.f);
  float sq[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    x[i] -= mean;
    sq[i & 3] += x[i] * x[i];
  }
  const float rstd = rsqrtf(quad_sum((sq[0] + sq[1]) + (sq[2] + sq[3])) * (1.f / 64.f) + 1e-5f);
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    const int at = 4 * (c & 1) + 16 * (c >> 1);
    const float4 ww = *reinterpret_cast<const float4*>(w + at), bb = *reinterpret_cast<const float4*>(bia + at);
    x[4 * c] = x[4 * c] * rstd * ww.x + bb.x;
    x[4 * c + 1] = x[4 * c + 1] * rstd * ww.y + bb.y;
    x[4 * c + 2] = x[4 * c + 2] * rstd * ww.z + bb.z;
    x[4 * c + 3] = x[4 * c + 3] * rstd * ww.w + bb.w;
  }
}

// cs: 3-D: cs[i] rotates the pair of elements 2i, 2i+1 of the sixteen; 2-D: cs[i] the elements i and i + 8.
template <int kMode>
__device__ __forceinline__ void rotate16(float (&x)[16], const float2 (&cs)[8]) {
  if constexpr (kMode == GCT_ROPE_NONE) return;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int lo = kMode == GCT_ROPE_2D ? i : 2 * i, hi = kMode == GCT_ROPE_2D ? i + 8 : 2 * i + 1;
    const float a = x[lo] * cs[i].x - x[hi] * cs[i].y;
    const float b = x[lo] * cs[i].y + x[hi] * cs[i].x;
    x[lo] = a;
    x[hi] = b;
  }
}

// kMode: rotation; kQkF32, kVF32: types of the sources of q and k, and of v.
template <int kMode, bool kQkF32, bool kVF32>
__global__ void __launch_bounds__(kPrepThreads) gct_prep_kernel(const PrepLaunch p) {
  __shared__ __align__(16) float s_norm[4][kHeadDim];       // q weight, q bias, k weight, k bias
  const int part = threadIdx.x & 3, e0 = 32 * (part >> 1) + 8 * (part & 1);
  const int rows = p.tokens * p.heads;
  const int row = (blockIdx.x * kPrepThreads + threadIdx.x) >> 2;
  const bool active = row < rows;           // inactive lanes (all four of a row) still take part in the shuffles
  const int r = active ? row : rows - 1;
  const int token = r / p.heads, h = r - token * p.heads;
  const bool do_q = p.q_src != nullptr && p.q_out != nullptr, do_kv = p.k_out != nullptr || p.pool != nullptr;
  const size_t src = static_cast<size_t>(token) * p.src_token_stride + static_cast<size_t>(h) * p.src_head_stride + e0;
  pdl_wait();
  RawRow<kQkF32> rq, rk;
  RawRow<kVF32> rv;
  if (do_q) rq.load(p.q_src, src);
  if (do_kv) {
    rk.load(p.k_src, src);
    rv.load(p.v_src, src);
  }
  // rotation coefficients of this lane
  float2 cs[8];
  if constexpr (kMode != GCT_ROPE_NONE) {
    const size_t entry = static_cast<size_t>(token % p.tokens_per_frame) * 32 + (kMode == GCT_ROPE_2D ? 16 * (part >> 1) + 8 * (part & 1) : e0 / 2);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const size_t at = 2 * (entry + (kMode == GCT_ROPE_2D ? 2 * i : 2 * (i & 1) + 8 * (i >> 1)));      // two entries
      if constexpr (kMode == kRope3dF64) {
        const double2* t = reinterpret_cast<const double2*>(static_cast<const double*>(p.rope_cs) + at);
        const double2 c0 = t[0], c1 = t[1];
        cs[2 * i] = make_float2(static_cast<float>(c0.x), static_cast<float>(c0.y));
        cs[2 * i + 1] = make_float2(static_cast<float>(c1.x), static_cast<float>(c1.y));
      } else {
        const float4 c = *reinterpret_cast<const float4*>(static_cast<const float*>(p.rope_cs) + at);
        cs[2 * i] = make_float2(c.x, c.y);
        cs[2 * i + 1] = make_float2(c.z, c.w);
      }
    }
  }
  // the running maximum as it was: older than the atomics below, so at worst one of them is issued in vain
  unsigned int seen = 0;
  if (do_kv && p.key_norm_max != nullptr) seen = *reinterpret_cast<volatile unsigned int*>(p.key_norm_max + h);
  // norm parameters, one element per array and thread of half a CTA
  {
    const int i = threadIdx.x & 63, which = threadIdx.x >> 6;
    const void* const w = which ? p.kn_w : p.qn_w;
    const void* const b = which ? p.kn_b : p.qn_b;
    if (w != nullptr) {
      s_norm[2 * which][i] = p.norm_dtype == GCT_F32 ? static_cast<const float*>(w)[i] : __bfloat162float(static_cast<const __nv_bfloat16*>(w)[i]);
      s_norm[2 * which + 1][i] = p.norm_dtype == GCT_F32 ? static_cast<const float*>(b)[i] : __bfloat162float(static_cast<const __nv_bfloat16*>(b)[i]);
    }
  }
  __syncthreads();

  // destination rows of K and V for this token
  __nv_bfloat16* k_row = nullptr;
  __nv_bfloat16* v_row = nullptr;
  if (p.k_out != nullptr) {
    k_row = p.k_out + static_cast<size_t>(token) * p.heads * kHeadDim;
    v_row = p.v_out + static_cast<size_t>(token) * p.heads * kHeadDim;
  } else if (p.pool != nullptr) {
    int page, slot;
    const int frame = token < p.tokens_per_frame ? 0 : token / p.tokens_per_frame, in_frame = token - frame * p.tokens_per_frame;
    const PageSlots& to = p.dst[frame];
    if (in_frame >= p.num_special) {
      page = to.patch_page;
      slot = in_frame - p.num_special;
    } else if (in_frame < to.sp_n0) {
      page = to.sp_page0;
      slot = to.sp_off0 + in_frame;
    } else {
      page = to.sp_page1;
      slot = in_frame - to.sp_n0;
    }
    if (page < 0 || page >= p.num_pages || slot < 0 || slot >= p.page_size) {
      if (active && part == 0) atomicCAS(p.status, 0, kStatusBadIndex);
    } else {
      const size_t page_elems = static_cast<size_t>(p.page_size) * p.heads * kHeadDim;
      k_row = p.pool + (static_cast<size_t>(page) * 2) * page_elems + static_cast<size_t>(slot) * p.heads * kHeadDim;
      v_row = k_row + page_elems;
    }
  }
  const bool in_range = !do_kv || k_row != nullptr;         // a token without a valid page writes nothing

  const size_t dst = static_cast<size_t>(h) * kHeadDim + e0;
  float x[16];
  if (do_q) {
    rq.floats(x);
    if (p.qn_w != nullptr) norm16(x, s_norm[0] + e0, s_norm[1] + e0);
    rotate16<kMode>(x, cs);
    if (active && in_range) store16(p.q_out + static_cast<size_t>(token) * p.heads * kHeadDim + dst, x);
  }
  if (do_kv) {
    rk.floats(x);
    if (p.kn_w != nullptr) norm16(x, s_norm[2] + e0, s_norm[3] + e0);
    rotate16<kMode>(x, cs);
    if (active && in_range) store16(k_row + dst, x);
    if (p.key_norm_max != nullptr) {
      // running maximum of |k| per head (an upper bound: fp32 values, inflated for the bf16 rounding).  Positive
      // floats order like their bit patterns; the look at the maximum above keeps atomics rare once it settles.
      float sq[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int i = 0; i < 16; ++i) sq[i & 3] += x[i] * x[i];
      const float nrm = sqrtf(quad_sum((sq[0] + sq[1]) + (sq[2] + sq[3]))) * 1.004f;
      if (active && in_range && part == 0 && !(nrm <= __uint_as_float(seen)))        // also taken for NaN
        atomicMax(reinterpret_cast<unsigned int*>(p.key_norm_max + h), nrm == nrm ? __float_as_uint(nrm) : 0x7f800000u);
    }
    rv.floats(x);
    if (active && in_range) store16(v_row + dst, x);
  }
}

// Eight consecutive elements as loaded, of either type: all loads of a thread are issued before the first conversion, which a
// branch on the type around load and conversion would prevent.
struct Raw8 {
  uint4 a, b;
  __device__ __forceinline__ void load(const void* base, int dtype, size_t elem) {
    const uint4* p = reinterpret_cast<const uint4*>(static_cast<const uint8_t*>(base) + elem * (dtype == GCT_F32 ? 4 : 2));
    a = p[0];
    if (dtype == GCT_F32) b = p[1];
  }
  __device__ __forceinline__ Row8 floats(int dtype) const {
    Row8 r;
    const uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
    if (dtype == GCT_F32) {
#pragma unroll
      for (int i = 0; i < 8; ++i) r.v[i] = __uint_as_float(w[i]);
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        r.v[2 * i] = __uint_as_float(w[i] << 16);
        r.v[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
      }
    }
    return r;
  }
};

// v = x + gamma * y per row, stored as sum_dtype (fp32 where x or gamma is, as the separate operations promote, else bf16), and
// LayerNorm(v) as bf16: the residual sums and norms of a block
// (lingbot_map/layers/block.py:217-310) in one pass over the row, which as separate tensor operations were four to
// six launches of 2-7 us each (scale, add, norm in fp32, cast to bf16 for the next Linear).
//
// A frame is 1005 rows of 1024 (6-12 MB), so the time is the chain load - mean - variance - store and how many rows are in
// flight.  Eight elements per thread and as many threads per row as that takes (whole warps; kThreads), everything the thread
// needs loaded first.  One warp per row, with the parameters fetched after the sums, took
// 5.6 us (norm alone), 9.2 us (sum and norm) and 6.4 us (sum alone), now 4.0, 4.8 and 3.6 us.
template <int kThreads>                   // threads per row: 32, 64, 128 or 256; columns <= 8 * kThreads
__global__ void __launch_bounds__(kThreads > 128 ? kThreads : 128) gct_residual_norm_kernel(const RowLaunch p) {
  constexpr int kRows = kThreads >= 128 ? 1 : 128 / kThreads, kWarps = kThreads / 32;      // rows per CTA, warps per row
  __shared__ float s_part[2][kRows][kWarps];
  pdl_wait();
  const int in_row = threadIdx.x % kThreads, local = threadIdx.x / kThreads, lane = threadIdx.x & 31, warp = in_row >> 5;
  const int64_t row = static_cast<int64_t>(blockIdx.x) * kRows + local;
  const int col = 8 * in_row;
  const bool active = row < p.rows && col < p.cols;
  const size_t at = static_cast<size_t>(row) * p.cols + col;
  const bool with_y = p.y != nullptr, with_gamma = with_y && p.gamma != nullptr, with_norm = p.norm_out != nullptr;
  Raw8 x, y, g, w, b;
  if (active) {
    x.load(p.x, p.x_dtype, at);
    if (with_y) y.load(p.y, GCT_BF16, at);
    if (with_gamma) g.load(p.gamma, p.gamma_dtype, col);
    if (with_norm) {
      w.load(p.norm_w, p.norm_dtype, col);
      b.load(p.norm_b, p.norm_dtype, col);
    }
  }
  Row8 v = {};
  if (active) {
    v = x.floats(p.x_dtype);
    if (with_y) {
      const Row8 yy = y.floats(GCT_BF16);
      if (with_gamma) {
        const Row8 gg = g.floats(p.gamma_dtype);
#pragma unroll
        for (int i = 0; i < 8; ++i) v.v[i] = fmaf(yy.v[i], gg.v[i], v.v[i]);
      } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) v.v[i] += yy.v[i];
      }
      if (p.sum_dtype == GCT_F32) {
        float4* d = reinterpret_cast<float4*>(static_cast<float*>(p.sum_out) + at);
        d[0] = make_float4(v.v[0], v.v[1], v.v[2], v.v[3]);
        d[1] = make_float4(v.v[4], v.v[5], v.v[6], v.v[7]);
      } else {
        store8(static_cast<__nv_bfloat16*>(p.sum_out) + at, v);
#pragma unroll
        for (int i = 0; i < 8; ++i) v.v[i] = __bfloat162float(__float2bfloat16_rn(v.v[i]));      // the norm is that of the stored sum
      }
    }
  }
  if (!with_norm) return;
  // sum over the threads of a row (idle ones add zero); every thread of the CTA comes here
  auto total = [&](float t, int step) -> float {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if constexpr (kWarps > 1) {
      if (lane == 0) s_part[step][local][warp] = t;
      __syncthreads();
      t = 0.f;
#pragma unroll
      for (int i = 0; i < kWarps; ++i) t += s_part[step][local][i];
    }
    return t;
  };
  float sum = 0.f, sq = 0.f;
#pragma unroll
  for (int i = 0; i < 8; ++i) sum += v.v[i];
  const float mean = total(sum, 0) / p.cols;
  if (active) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      v.v[i] -= mean;
      sq = fmaf(v.v[i], v.v[i], sq);
    }
  }
  const float rstd = rsqrtf(total(sq, 1) / p.cols + p.eps);
  if (!active) return;
  const Row8 ww = w.floats(p.norm_dtype), bb = b.floats(p.norm_dtype);
  Row8 r;
#pragma unroll
  for (int i = 0; i < 8; ++i) r.v[i] = fmaf(v.v[i] * rstd, ww.v[i], bb.v[i]);
  store8(p.norm_out + at, r);
}

// x = 0.5 x (1 + erf(x / sqrt 2)) of bf16 values in place, in fp32: the activation between the two Linear layers of a block.  A frame is
// 1005 x 4096 values (8 MB, just written: they lie in L2), so the time is the launch, which overlaps the end of the product before,
// and one round trip.  In place of a tensor operation (6.5 us, out of place, and its dispatch), together with the appends of a scale
// pass in one launch: a sequence's first sixteen frames through two layer pairs 3668 -> 3617 us.
__global__ void __launch_bounds__(256) gct_gelu_kernel(__nv_bfloat16* __restrict__ x, int64_t n) {
  pdl_wait();
  auto gelu = [](float v) { return 0.5f * v * (1.f + erff(v * 0.70710678118654752f)); };
  const int64_t i = (static_cast<int64_t>(blockIdx.x) * 256 + threadIdx.x) * 8;
  if (i + 8 <= n) {
    Row8 r = load8(x, GCT_BF16, i);
#pragma unroll
    for (int e = 0; e < 8; ++e) r.v[e] = gelu(r.v[e]);
    store8(x + i, r);
  } else {
    for (int64_t e = i; e < n; ++e) x[e] = __float2bfloat16_rn(gelu(__bfloat162float(x[e])));
  }
}

// cos/sin table of the 2-D rotation from integer (y, x) positions [tokens, 2] (lingbot_map/layers/rope.py:105-119): entry
// 16 * axis + j is the angle position * base^(-2j/32) in fp32.
__global__ void gct_rope2d_positions_kernel(const int64_t* __restrict__ pos, int64_t token_stride, int64_t axis_stride, int tokens, float base,
                                            float* __restrict__ cs) {
  pdl_wait();
  const int idx = blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= tokens * 32) return;
  const int token = idx >> 5, axis = (idx >> 4) & 1, j = idx & 15;
  const float inv = 1.0f / powf(base, static_cast<float>(2 * j) / 32.0f);
  const float ang = static_cast<float>(pos[token * token_stride + axis * axis_stride]) * inv;
  float sn, cn;
  sincosf(ang, &sn, &cn);
  *reinterpret_cast<float2*>(cs + 2 * idx) = make_float2(cn, sn);
}

__global__ void gct_cast_kernel(const float* __restrict__ src, __nv_bfloat16* __restrict__ dst, int64_t n4) {
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n4; i += stride) {
    const float4 v = reinterpret_cast<const float4*>(src)[i];
    __nv_bfloat162 a = __floats2bfloat162_rn(v.x, v.y), b = __floats2bfloat162_rn(v.z, v.w);
    uint2 w;
    w.x = *reinterpret_cast<uint32_t*>(&a);
    w.y = *reinterpret_cast<uint32_t*>(&b);
    reinterpret_cast<uint2*>(dst)[i] = w;
  }
}

// out = sum_g w_g O_g / sum_g w_g,  w_g = exp(lse_g - max_g lse_g) per (query, head) row.
//
// Eight lanes per row, eight consecutive elements each.  The partials were just written and mostly lie in L2, so the time is
// round trips: four groups are in flight per lane from the start, under the look at the log-sum-exps, and the next four while
// these are added up.  One warp per row with one 8-byte load in flight after the log-sum-exps took 8.9 us for three
// groups and 14.0 us for nine (1005 x 16 rows, cold L2), now 8.0 and 11.1 us.
// kWide: 16-byte accesses; else (a base or group stride that is only a multiple of two floats) 8-byte ones.
template <bool kWide>
__global__ void __launch_bounds__(128)
gct_merge_kernel(const float* __restrict__ parts, const float* __restrict__ lse, int groups, int64_t rows,
                 int64_t parts_stride, int64_t lse_stride, __nv_bfloat16* __restrict__ out_bf16,
                 float* __restrict__ out_f32, float* __restrict__ lse_out) {
  constexpr int kBatch = 4;
  pdl_wait();
  const int part = threadIdx.x & 7;
  const int64_t row = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 3;
  if (row >= rows) return;
  const float* src = parts + row * kHeadDim + 8 * part;
  auto load = [&](int g0, Row8(&o)[kBatch]) {
#pragma unroll
    for (int u = 0; u < kBatch; ++u) {
      if (g0 + u >= groups) continue;
      const float* p = src + static_cast<int64_t>(g0 + u) * parts_stride;
      if constexpr (kWide) {
        o[u] = load8(p, GCT_F32, 0);
      } else {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float2 f = *reinterpret_cast<const float2*>(p + 2 * i);
          o[u].v[2 * i] = f.x;
          o[u].v[2 * i + 1] = f.y;
        }
      }
    }
  };
  Row8 o0[kBatch], o1[kBatch];
  load(0, o0);
  const float* l = lse + row;
  float mx = -INFINITY;
#pragma unroll 8
  for (int g = 0; g < groups; ++g) mx = fmaxf(mx, l[static_cast<int64_t>(g) * lse_stride]);
  float den = 0.f;
  Row8 acc = {};
  auto add = [&](int g0, const Row8(&o)[kBatch]) {
#pragma unroll
    for (int u = 0; u < kBatch; ++u) {
      if (g0 + u >= groups) continue;
      const float w = __expf(l[static_cast<int64_t>(g0 + u) * lse_stride] - mx);
#pragma unroll
      for (int i = 0; i < 8; ++i) acc.v[i] = fmaf(w, o[u].v[i], acc.v[i]);
      den += w;
    }
  };
  for (int g = 0; g < groups; g += 2 * kBatch) {
    load(g + kBatch, o1);
    add(g, o0);
    load(g + 2 * kBatch, o0);
    add(g + kBatch, o1);
  }
  const float inv = 1.f / den;
#pragma unroll
  for (int i = 0; i < 8; ++i) acc.v[i] *= inv;
  const int64_t dst = row * kHeadDim + 8 * part;
  if (out_bf16 != nullptr) {
    if constexpr (kWide) {
      store8(out_bf16 + dst, acc);
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i) *reinterpret_cast<__nv_bfloat162*>(out_bf16 + dst + 2 * i) = __floats2bfloat162_rn(acc.v[2 * i], acc.v[2 * i + 1]);
    }
  }
  if (out_f32 != nullptr) {
#pragma unroll
    for (int i = 0; i < 4; ++i) *reinterpret_cast<float2*>(out_f32 + dst + 2 * i) = make_float2(acc.v[2 * i], acc.v[2 * i + 1]);
  }
  if (lse_out != nullptr && part == 0) lse_out[row] = mx + logf(den);
}

// Eight lanes per K row of the pool (16 bytes each), four rows per warp and load, four loads in flight per lane.
__global__ void __launch_bounds__(256)
gct_scan_keys_kernel(const __nv_bfloat16* __restrict__ pool, int64_t total_rows, int page_size, int heads,
                     float* key_norm_max) {
  const int lane = threadIdx.x & 31, part = lane & 7, sub = lane >> 3;
  const int64_t warps = (static_cast<int64_t>(gridDim.x) * blockDim.x) >> 5;
  const int64_t rows_per_page = static_cast<int64_t>(page_size) * heads;
  constexpr int kUnroll = 4;
  for (int64_t base = ((static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5) * (4 * kUnroll);
       base < total_rows; base += warps * (4 * kUnroll)) {
    uint4 v[kUnroll];
    int head[kUnroll];
#pragma unroll
    for (int u = 0; u < kUnroll; ++u) {
      const int64_t r = base + 4 * u + sub;
      const int64_t rr = r < total_rows ? r : total_rows - 1;          // tail: repeat the last row
      const int64_t page = rr / rows_per_page, in_page = rr - page * rows_per_page;
      head[u] = static_cast<int>(in_page % heads);
      v[u] = *reinterpret_cast<const uint4*>(pool + (page * 2 * rows_per_page + in_page) * kHeadDim + 8 * part);
    }
#pragma unroll
    for (int u = 0; u < kUnroll; ++u) {
      const uint32_t w[4] = {v[u].x, v[u].y, v[u].z, v[u].w};
      float sq = 0.f;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w[i]));
        sq += f.x * f.x + f.y * f.y;
      }
      sq = row_sum(sq);
      if (part == 0) {
        const float nrm = sqrtf(sq);
        unsigned int* slot = reinterpret_cast<unsigned int*>(key_norm_max + head[u]);
        if (!(nrm <= __uint_as_float(*reinterpret_cast<volatile unsigned int*>(slot))))
          atomicMax(slot, nrm == nrm ? __float_as_uint(nrm) : 0x7f800000u);
      }
    }
  }
}

// cs[token][m] = (cos, sin) of the m-th complex frequency; fp64 angles as the reference's table
// (lingbot_map/layers/rope.py:326-334,399-413): m<10 time (dim 20), m<21 height (dim 22), else width (dim 22).
__global__ void gct_rope3d_table_kernel(int f, int pph, int ppw, int ns, float* cs) {
  pdl_wait();
  const int idx = blockIdx.x * blockDim.x + threadIdx.x;
  const int tokens = ns + pph * ppw;
  if (idx >= tokens * 32) return;
  const int token = idx >> 5, m = idx & 31;
  int ph, pw;
  if (token < ns) {
    ph = pw = token;
  } else {
    const int pidx = token - ns;
    ph = ns + pidx / ppw;
    pw = ns + pidx % ppw;
  }
  double pos, expo;
  if (m < 10) {
    pos = f;
    expo = (2.0 * m) / 20.0;
  } else if (m < 21) {
    pos = ph;
    expo = (2.0 * (m - 10)) / 22.0;
  } else {
    pos = pw;
    expo = (2.0 * (m - 21)) / 22.0;
  }
  const double ang = pos * (1.0 / pow(10000.0, expo));
  cs[2 * idx] = static_cast<float>(cos(ang));
  cs[2 * idx + 1] = static_cast<float>(sin(ang));
}

// 2-D table (lingbot_map/layers/rope.py:105-119; positions lingbot_map/aggregator/base.py:436-440):
// entry 16*axis + j holds the angle pos_axis * base^(-2j/32), computed in fp32 like the reference.
__global__ void gct_rope2d_table_kernel(int pph, int ppw, int ns, float base, float* cs) {
  const int idx = blockIdx.x * blockDim.x + threadIdx.x;
  const int tokens = ns + pph * ppw;
  if (idx >= tokens * 32) return;
  const int token = idx >> 5, e = idx & 31;
  const int axis = e >> 4, j = e & 15;
  int pos = 0;
  if (token >= ns) {
    const int pidx = token - ns;
    pos = (axis == 0 ? pidx / ppw : pidx % ppw) + 1;
  }
  const float inv = 1.0f / powf(base, static_cast<float>(2 * j) / 32.0f);
  const float ang = static_cast<float>(pos) * inv;
  cs[2 * idx] = cosf(ang);
  cs[2 * idx + 1] = sinf(ang);
}

}  // namespace

int launch_prep(const PrepLaunch& p, cudaStream_t stream) {
  if (p.tokens <= 0 || p.heads <= 0 || p.tokens_per_frame <= 0) return fail(GCT_ERR_INVALID, "prep: bad shape");
  if (p.rope_mode != GCT_ROPE_NONE && p.rope_cs == nullptr) return fail(GCT_ERR_INVALID, "prep: rope table missing");
  if (p.rope_mode == GCT_ROPE_2D && p.rope_f64) return fail(GCT_ERR_INVALID, "prep: the 2-D table is float");
  if ((p.src_token_stride | p.src_head_stride) & 7)
    return fail(GCT_ERR_INVALID, "prep: source strides must be multiples of 8 elements (16-byte vector loads)");
  auto misaligned = [](const void* q) { return q != nullptr && (reinterpret_cast<uintptr_t>(q) & 15) != 0; };
  if (misaligned(p.q_src) || misaligned(p.k_src) || misaligned(p.v_src) || misaligned(p.q_out) || misaligned(p.k_out) ||
      misaligned(p.v_out) || misaligned(p.pool) || misaligned(p.qn_w) || misaligned(p.qn_b) || misaligned(p.kn_w) ||
      misaligned(p.kn_b) || misaligned(p.rope_cs))
    return fail(GCT_ERR_INVALID, "prep: tensors must be 16-byte aligned");
  if (p.k_out == nullptr && p.pool != nullptr && p.tokens > static_cast<long long>(kAppendFrames) * p.tokens_per_frame)
    return fail(GCT_ERR_INVALID, "prep: more frames than one launch takes");
  const long long rows = static_cast<long long>(p.tokens) * p.heads;
  if (rows > (1ll << 28)) return fail(GCT_ERR_INVALID, "prep: too many rows");
  const dim3 grid(static_cast<unsigned>((rows * 4 + kPrepThreads - 1) / kPrepThreads)), block(kPrepThreads);
  const bool qk32 = p.src_dtype_qk == GCT_F32, v32 = p.src_dtype_v == GCT_F32;
  auto pick = [&](auto mode) {
    constexpr int m = decltype(mode)::value;
    return qk32 ? (v32 ? gct_prep_kernel<m, true, true> : gct_prep_kernel<m, true, false>)
                : (v32 ? gct_prep_kernel<m, false, true> : gct_prep_kernel<m, false, false>);
  };
  auto kernel = p.rope_mode == GCT_ROPE_3D ? (p.rope_f64 ? pick(std::integral_constant<int, kRope3dF64>()) : pick(std::integral_constant<int, GCT_ROPE_3D>()))
                : p.rope_mode == GCT_ROPE_2D ? pick(std::integral_constant<int, GCT_ROPE_2D>())
                                             : pick(std::integral_constant<int, GCT_ROPE_NONE>());
  GCT_CUDA_CHECK(launch_pdl(kernel, grid, block, 0, stream, p));
  return GCT_OK;
}

int launch_residual_norm(const RowLaunch& p, cudaStream_t stream) {
  if (p.rows <= 0 || p.cols <= 0 || p.cols % 8 != 0 || p.cols > kRowMaxCols) return fail(GCT_ERR_INVALID, "residual norm: bad shape");
  auto misaligned = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15) != 0; };
  if (misaligned(p.x) || misaligned(p.y) || misaligned(p.gamma) || misaligned(p.norm_w) || misaligned(p.norm_b) || misaligned(p.sum_out) ||
      misaligned(p.norm_out))
    return fail(GCT_ERR_INVALID, "residual norm: tensors must be 16-byte aligned");
  // threads per row: eight columns each, whole warps; short rows share a CTA of 128
  const int threads = p.cols <= 256 ? 32 : p.cols <= 512 ? 64 : p.cols <= 1024 ? 128 : 256;
  const int64_t rows_per_cta = threads >= 128 ? 1 : 128 / threads, ctas = (p.rows + rows_per_cta - 1) / rows_per_cta;
  if (ctas > 0x7fffffff) return fail(GCT_ERR_INVALID, "residual norm: too many rows");
  const dim3 grid(static_cast<unsigned>(ctas)), block(threads > 128 ? threads : 128);
  auto kernel = threads == 32 ? gct_residual_norm_kernel<32> : threads == 64 ? gct_residual_norm_kernel<64>
                : threads == 128 ? gct_residual_norm_kernel<128> : gct_residual_norm_kernel<256>;
  GCT_CUDA_CHECK(launch_pdl(kernel, grid, block, 0, stream, p));
  return GCT_OK;
}

int launch_gelu(__nv_bfloat16* x, int64_t n, cudaStream_t stream) {
  const int64_t ctas = (n + 2047) / 2048;
  if (n < 0 || ctas > 0x7fffffff || (reinterpret_cast<uintptr_t>(x) & 15) != 0) return fail(GCT_ERR_INVALID, "gelu: bad argument");
  if (n == 0) return GCT_OK;
  GCT_CUDA_CHECK(launch_pdl(gct_gelu_kernel, dim3(static_cast<unsigned>(ctas)), dim3(256), 0, stream, x, n));
  return GCT_OK;
}

int launch_rope2d_positions(const int64_t* pos, int64_t token_stride, int64_t axis_stride, int tokens, float base, float* cs, cudaStream_t stream) {
  const dim3 grid((tokens * 32 + 255) / 256), block(256);
  GCT_CUDA_CHECK(launch_pdl(gct_rope2d_positions_kernel, grid, block, 0, stream, pos, token_stride, axis_stride, tokens, base, cs));
  return GCT_OK;
}

int launch_cast_bf16(const float* src, __nv_bfloat16* dst, int64_t n, cudaStream_t stream) {
  if (n % 4 != 0) return fail(GCT_ERR_INVALID, "cast: element count must be a multiple of 4");
  const int64_t n4 = n / 4;
  const int blocks = static_cast<int>(n4 / 256 + 1 < 1184 ? n4 / 256 + 1 : 1184);
  gct_cast_kernel<<<blocks, 256, 0, stream>>>(src, dst, n4);
  GCT_CUDA_CHECK(cudaGetLastError());
  return GCT_OK;
}

int launch_merge(const float* parts, const float* lse, int groups, int64_t rows, __nv_bfloat16* out_bf16,
                 float* out_f32, float* lse_out, cudaStream_t stream, int64_t parts_stride, int64_t lse_stride) {
  if (groups <= 0 || rows <= 0) return fail(GCT_ERR_INVALID, "merge: bad shape");
  if (parts_stride <= 0) parts_stride = rows * kHeadDim;
  if (lse_stride <= 0) lse_stride = rows;
  if (parts_stride % 2 != 0) return fail(GCT_ERR_INVALID, "merge: group stride of the partial outputs must be even");
  const int64_t blocks = (rows * 8 + 127) / 128;
  if (blocks > 0x7fffffff) return fail(GCT_ERR_INVALID, "merge: too many rows");
  const bool wide = parts_stride % 4 == 0 && ((reinterpret_cast<uintptr_t>(parts) | reinterpret_cast<uintptr_t>(out_bf16)) & 15) == 0;
  GCT_CUDA_CHECK(launch_pdl(wide ? gct_merge_kernel<true> : gct_merge_kernel<false>, dim3(static_cast<unsigned>(blocks)), dim3(128), 0, stream, parts,
                            lse, groups, rows, parts_stride, lse_stride, out_bf16, out_f32, lse_out));
  return GCT_OK;
}

int launch_scan_keys(const __nv_bfloat16* pool, int num_pages, int page_size, int heads, float* key_norm_max,
                     cudaStream_t stream) {
  if (pool == nullptr || key_norm_max == nullptr || num_pages <= 0 || page_size <= 0 || heads <= 0)
    return fail(GCT_ERR_INVALID, "scan_keys: bad argument");
  GCT_CUDA_CHECK(cudaMemsetAsync(key_norm_max, 0, static_cast<size_t>(heads) * sizeof(float), stream));
  const int64_t total_rows = static_cast<int64_t>(num_pages) * page_size * heads;
  gct_scan_keys_kernel<<<148 * 8, 256, 0, stream>>>(pool, total_rows, page_size, heads, key_norm_max);
  GCT_CUDA_CHECK(cudaGetLastError());
  return GCT_OK;
}

int launch_rope3d_table(int f, int pph, int ppw, int ns, float* cs, cudaStream_t stream) {
  const int n = (ns + pph * ppw) * 32;
  GCT_CUDA_CHECK(launch_pdl(gct_rope3d_table_kernel, dim3((n + 255) / 256), dim3(256), 0, stream, f, pph, ppw, ns, cs));
  return GCT_OK;
}

int launch_rope2d_table(int pph, int ppw, int ns, float base, float* cs, cudaStream_t stream) {
  const int n = (ns + pph * ppw) * 32;
  gct_rope2d_table_kernel<<<(n + 255) / 256, 256, 0, stream>>>(pph, ppw, ns, base, cs);
  GCT_CUDA_CHECK(cudaGetLastError());
  return GCT_OK;
}

}  // namespace gct

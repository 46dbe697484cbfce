// Point-cloud helpers of the offline renderer as plain CUDA: frustum culling and Morton voxelisation.
//
// Restates demo_render/render_cuda_ext/frustum_cull/frustum_cull.cu:5-33 and
// demo_render/render_cuda_ext/voxel_morton/voxel_morton.cu:5-62 of the reference (compute only; the renderer that
// consumes them needs a graphics API and is not part of this library).  Both are streams over AoS xyz floats:
// 13 B per point (cull: HBM bound, the kernel alone 19.7 us for 8 M points = 5.3 TB/s) and 24 B read + 44 B written per point (voxelise).
// Arithmetic is written with explicitly rounded single operations (no fused multiply-add, IEEE division), so that
// a float32 CPU restatement reproduces every mask bit and every Morton code exactly.
#include <algorithm>
#include <chrono>

#include "gct_common.h"

namespace gct {
namespace {

struct CullArgs {
  float R[9], t[3];
  const float* R_dev;      // not null: the rotation and translation are in device memory
  const float* t_dev;
  int R_row, R_col, t_step;   // their strides
  float fx, fy, cx, cy, near_plane, far_plane;
  int W, H;
  float mid_u, mid_v, in_u, in_v, out_u, out_v;      // the test without divisions
  bool depth_tame;
};

__device__ __forceinline__ float camera_axis(const CullArgs& a, int row, float x, float y, float z) {
  return __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(a.R[3 * row], x), __fmul_rn(a.R[3 * row + 1], y)), __fmul_rn(a.R[3 * row + 2], z)), a.t[row]);
}

// The mask as it is defined: pixel coordinates by IEEE division.
__device__ bool cull_exact(float x, float y, float z, const CullArgs& a) {
  const float px = camera_axis(a, 0, x, y, z), py = camera_axis(a, 1, x, y, z), pz = camera_axis(a, 2, x, y, z);
  if (pz <= a.near_plane || pz >= a.far_plane) return false;            // frustum_cull.cu:25-28 (NaN depth: kept there too)
  const float fu = __fadd_rn(__fmul_rn(__fdiv_rn(px, pz), a.fx), a.cx);
  const float fv = __fadd_rn(__fmul_rn(__fdiv_rn(py, pz), a.fy), a.cy);
  // (int) of a float outside the int range is undefined in C; such points are outside every image
  if (!(fu > -2147483648.f && fu < 2147483648.f && fv > -2147483648.f && fv < 2147483648.f)) return false;
  const int u = static_cast<int>(fu), v = static_cast<int>(fv);       // truncation toward zero, as the reference
  return u >= 0 && u < a.W && v >= 0 && v < a.H;
}

// Most points without a division.  An image of size >= 1 is the open interval (-1, size) per axis (truncation maps (-1, 0] to pixel 0;
// an empty one has no such interval, and the host sets the limits so that every point is out);
// with the coordinate taken from its middle, |px / pz * f + (c - mid)| against half its width decides.  The product with an
// approximate reciprocal is off by less than 2^-20 relative, which near a border is less than 2^-20 (|c| + size + 1);
// in_ and out_ keep ten times that away from the border.  In between, and for anything not finite, `undecided` is set.
__device__ __forceinline__ bool cull_fast(float x, float y, float z, const CullArgs& a, bool& undecided) {
  const float px = camera_axis(a, 0, x, y, z), py = camera_axis(a, 1, x, y, z), pz = camera_axis(a, 2, x, y, z);
  if (pz <= a.near_plane || pz >= a.far_plane) return false;
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(pz));
  const float u = fabsf(fmaf(px * r, a.fx, a.mid_u)), v = fabsf(fmaf(py * r, a.fy, a.mid_v));
  const bool tame = a.depth_tame || (fabsf(pz) > 1e-30f && fabsf(pz) < 1e30f);      // the reciprocal neither flushes nor overflows
  const bool in = u < a.in_u && v < a.in_v, out = u > a.out_u || v > a.out_v;
  undecided = !(tame && (in || out));
  return in;
}

// A thread takes four points = three 16-byte loads and has the next four on their way.  The kernel alone with two IEEE divisions
// per point and one load in flight: 22.5 us at 8 M points; this way 19.7 us (16 us at the measured copy rate; as one call
// among others, with its launch and the allocation of the mask, 22.6 us, and 21.1 us since the launch overlaps the end of the kernel before;
// behind an elementwise kernel of the tensor library the pair 33.9 -> 32.7 us).
__global__ void __launch_bounds__(256) gct_frustum_cull_kernel(const float* __restrict__ pts, CullArgs a, uint8_t* __restrict__ visible,
                                                               int64_t n) {
  pdl_wait();
  if (a.R_dev != nullptr) {
#pragma unroll
    for (int i = 0; i < 9; ++i) a.R[i] = __ldg(a.R_dev + (i / 3) * a.R_row + (i % 3) * a.R_col);
#pragma unroll
    for (int i = 0; i < 3; ++i) a.t[i] = __ldg(a.t_dev + i * a.t_step);
  }
  const int64_t quads = n / 4;
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  auto load = [&](int64_t qd, float4(&v)[3]) {
    const float4* p = reinterpret_cast<const float4*>(pts) + 3 * qd;
    v[0] = p[0];                                                       // x0 y0 z0 x1 | y1 z1 x2 y2 | z2 x3 y3 z3
    v[1] = p[1];
    v[2] = p[2];
  };
  auto test = [&](int64_t qd, const float4(&v)[3]) {
    bool d0 = false, d1 = false, d2 = false, d3 = false;
    uchar4 m;
    m.x = cull_fast(v[0].x, v[0].y, v[0].z, a, d0);
    m.y = cull_fast(v[0].w, v[1].x, v[1].y, a, d1);
    m.z = cull_fast(v[1].z, v[1].w, v[2].x, a, d2);
    m.w = cull_fast(v[2].y, v[2].z, v[2].w, a, d3);
    if (d0 || d1 || d2 || d3) {
      m.x = cull_exact(v[0].x, v[0].y, v[0].z, a);
      m.y = cull_exact(v[0].w, v[1].x, v[1].y, a);
      m.z = cull_exact(v[1].z, v[1].w, v[2].x, a);
      m.w = cull_exact(v[2].y, v[2].z, v[2].w, a);
    }
    reinterpret_cast<uchar4*>(visible)[qd] = m;
  };
  float4 v0[3], v1[3];
  int64_t qd = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (qd < quads) load(qd, v0);
  for (; qd < quads; qd += 2 * stride) {
    if (qd + stride < quads) load(qd + stride, v1);
    test(qd, v0);
    if (qd + stride >= quads) break;
    if (qd + 2 * stride < quads) load(qd + 2 * stride, v0);
    test(qd + stride, v1);
  }
  if (blockIdx.x == 0 && threadIdx.x < n - 4 * quads) {
    const int64_t i = 4 * quads + threadIdx.x;
    visible[i] = cull_exact(pts[3 * i], pts[3 * i + 1], pts[3 * i + 2], a);
  }
}

// Interleave the low 21 bits of x, y, z (voxel_morton.cu:5-18).
__device__ __forceinline__ uint64_t expand_bits(uint64_t v) {
  v = (v | (v << 32)) & 0x1f00000000ffffULL;
  v = (v | (v << 16)) & 0x1f0000ff0000ffULL;
  v = (v | (v << 8)) & 0x100f00f00f00f00fULL;
  v = (v | (v << 4)) & 0x10c30c30c30c30c3ULL;
  v = (v | (v << 2)) & 0x1249249249249249ULL;
  return v;
}

__global__ void __launch_bounds__(256) gct_voxel_morton_kernel(const float* __restrict__ xyz, const float* __restrict__ rgb,
                                                               float voxel_size, int64_t n, int64_t* __restrict__ codes,
                                                               float* __restrict__ centers, float* __restrict__ colors) {
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride) {
    const float x = xyz[3 * i], y = xyz[3 * i + 1], z = xyz[3 * i + 2];
    const int ix = static_cast<int>(floorf(__fdiv_rn(x, voxel_size)));
    const int iy = static_cast<int>(floorf(__fdiv_rn(y, voxel_size)));
    const int iz = static_cast<int>(floorf(__fdiv_rn(z, voxel_size)));
    constexpr int kOffset = 1 << 20;                                   // voxel_morton.cu:36-38
    const uint64_t code = expand_bits(static_cast<uint64_t>(static_cast<uint32_t>(ix + kOffset))) |
                          (expand_bits(static_cast<uint64_t>(static_cast<uint32_t>(iy + kOffset))) << 1) |
                          (expand_bits(static_cast<uint64_t>(static_cast<uint32_t>(iz + kOffset))) << 2);
    codes[i] = static_cast<int64_t>(code);
    centers[3 * i] = __fmul_rn(__fadd_rn(static_cast<float>(ix), 0.5f), voxel_size);
    centers[3 * i + 1] = __fmul_rn(__fadd_rn(static_cast<float>(iy), 0.5f), voxel_size);
    centers[3 * i + 2] = __fmul_rn(__fadd_rn(static_cast<float>(iz), 0.5f), voxel_size);
    colors[3 * i] = rgb[3 * i];
    colors[3 * i + 1] = rgb[3 * i + 1];
    colors[3 * i + 2] = rgb[3 * i + 2];
  }
}

__global__ void __launch_bounds__(256) gct_mark_unique_kernel(const int64_t* __restrict__ sorted, int64_t n, uint8_t* __restrict__ mask) {
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride)
    mask[i] = (i == 0) || (sorted[i] != sorted[i - 1]);                // voxel_morton.cu:49-62
}

// ---- voxelisation of a cloud of up to kVoxelMaxPoints points: codes, stable sort, first point of each voxel ----
//
// A frame's cloud is small (about 200 k points, 2.4 MB), so the time is launches and passes, not bandwidth: a general
// 64-bit sort made eight radix passes over (code, index), then two gathers, a mark, a compaction and three more gathers
// (34 launches, 240 us).  Voxel indices within +-2^nb only need a Morton key of 3 (nb + 1) bits (bits nb ... 20 of an offset
// index all equal the complement of its sign, so leaving them out does not change the order): 24-33 bits for a room at
// centimetres, four or five passes of eight bits.  The number of bits is found on the device, so the host waits only once, for
// the number of voxels.  Measured for 196 k points: 240 us, as short-key passes 68 us, with the passes in one launch 53 us.
constexpr int kVoxelTile = 2048;                 // keys per CTA of a pass: a frame's cloud makes about one CTA per SM
constexpr int kVoxelThreads = 512;
constexpr int kVoxelWarps = kVoxelThreads / 32;
constexpr int kVoxelPerThread = kVoxelTile / kVoxelThreads;
constexpr int kVoxelMaxTiles = 256;              // every CTA of a pass adds up the digit counts of all tiles
constexpr int kVoxelMaxPasses = 8;
constexpr int kVoxelOffset = 1 << 20;            // voxel_morton.cu:36-38
constexpr int32_t kVoxelPending = -1, kVoxelFailed = -2;      // in place of a tile's count
constexpr std::chrono::microseconds kVoxelLook{150};          // the largest cloud of the sort: up to 126 us from the call to its counts

struct VoxelScratch {
  uint64_t* keys0;         // Morton codes and indices, two buffers
  uint64_t* keys1;
  uint32_t* index0;
  uint32_t* index1;
  uint32_t* extent;        // [tiles] OR of the index magnitudes of a tile
  uint32_t* hist;          // [passes][tiles][256] digit counts
  int32_t* heads;          // [tiles] first points of voxels in a tile of the sorted keys
  uint32_t* arrived;       // CTAs that have come to the barriers of the sort, all barriers together
  int n, tiles;
  __device__ __forceinline__ uint64_t* keys(int i) const { return i & 1 ? keys1 : keys0; }
  __device__ __forceinline__ uint32_t* index(int i) const { return i & 1 ? index1 : index0; }
};

__device__ __forceinline__ int voxel_index(float p, float voxel_size) { return static_cast<int>(floorf(__fdiv_rn(p, voxel_size))); }
// The index as the Morton code sees it: its low 21 bits after the offset, centred again.
__device__ __forceinline__ int voxel_wrapped(int i) {
  return static_cast<int>((static_cast<uint32_t>(i) + static_cast<uint32_t>(kVoxelOffset)) & 0x1fffffu) - kVoxelOffset;
}
__device__ __forceinline__ uint64_t morton(uint32_t x, uint32_t y, uint32_t z) {
  return expand_bits(x) | (expand_bits(y) << 1) | (expand_bits(z) << 2);
}

// Key bits per axis without the sign, from the tiles' extents (a warp's worth of loads); at least three, so that the first
// digit is the low byte of the code whatever the extent.
__device__ __forceinline__ int voxel_axis_bits(const VoxelScratch& s) {
  uint32_t m = 0;
  for (int t = threadIdx.x & 31; t < s.tiles; t += 32) m |= s.extent[t];
  m = __reduce_or_sync(0xffffffffu, m);
  return max(3, 32 - __clz(m));
}
__host__ __device__ __forceinline__ int voxel_passes(int axis_bits) { return (3 * (axis_bits + 1) + 7) / 8; }
// The key of a code: 3 * axis_bits low bits and the three signs above them.
__device__ __forceinline__ uint64_t voxel_key(uint64_t code, int axis_bits) {
  return (code & ((1ull << (3 * axis_bits)) - 1)) | (code >> 60 << (3 * axis_bits));
}

__global__ void __launch_bounds__(kVoxelThreads) gct_voxel_code_kernel(const float* __restrict__ xyz, float voxel_size, VoxelScratch s) {
  pdl_wait();
  __shared__ uint32_t s_hist[256];
  __shared__ uint32_t s_or;
  if (threadIdx.x < 256) s_hist[threadIdx.x] = 0;
  if (threadIdx.x == 0) s_or = 0;
  __syncthreads();
  uint32_t m = 0;
#pragma unroll
  for (int u = 0; u < kVoxelPerThread; ++u) {
    const int i = blockIdx.x * kVoxelTile + u * kVoxelThreads + threadIdx.x;
    if (i < s.n) {
      uint32_t w[3];
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const int v = voxel_wrapped(voxel_index(xyz[3 * i + c], voxel_size));
        m |= static_cast<uint32_t>(v ^ (v >> 31));
        w[c] = static_cast<uint32_t>(v + kVoxelOffset);
      }
      const uint64_t code = morton(w[0], w[1], w[2]);
      s.keys0[i] = code;
      s.index0[i] = static_cast<uint32_t>(i);
      atomicAdd(&s_hist[code & 255], 1u);
    }
  }
  m = __reduce_or_sync(0xffffffffu, m);
  if ((threadIdx.x & 31) == 0) atomicOr(&s_or, m);
  __syncthreads();
  if (threadIdx.x == 0) s.extent[blockIdx.x] = s_or;
  if (blockIdx.x == 0 && threadIdx.x == 0) *s.arrived = 0;
  uint32_t* hist = s.hist + static_cast<size_t>(blockIdx.x) * 256;
  for (int k = threadIdx.x; k < kVoxelMaxPasses * 256; k += kVoxelThreads)      // counts of the later passes start from zero
    hist[static_cast<size_t>(k >> 8) * s.tiles * 256 + (k & 255)] = k < 256 ? s_hist[k] : 0u;
}

struct VoxelShared {
  uint32_t warp[kVoxelWarps][256];
  uint32_t total[256], before[256];
  uint32_t global[256];                         // first global position of a digit of this tile, minus its first local one
  uint32_t scan[2][8];
  uint64_t code[kVoxelTile];
  uint32_t index[kVoxelTile];
  int met;
};

// One stable pass over 8 bits of one tile.  A warp owns 128 consecutive keys of the tile and ranks them 32 at a time (one ballot per
// digit bit); the tile's base per digit is the number of smaller digits anywhere plus the number of equal ones in earlier
// tiles.  While scattering, the digit counts of the next pass are gathered by the destination tile.  What other CTAs wrote in an
// earlier pass is read past L1, which may hold lines of the pass before.
__device__ __forceinline__ void voxel_pass(int pass, int passes, int tile, int axis_bits, const VoxelScratch& s, VoxelShared& sh) {
  auto& s_warp = sh.warp;
  auto& s_total = sh.total;
  auto& s_before = sh.before;
  auto& s_global = sh.global;
  auto& s_scan = sh.scan;
  auto& s_code = sh.code;
  auto& s_index = sh.index;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, shift = 8 * pass;
  const uint64_t* keys = s.keys(pass);
  const uint32_t* index = s.index(pass);
  uint64_t code[kVoxelPerThread];
  uint32_t idx[kVoxelPerThread], rank[kVoxelPerThread];
#pragma unroll
  for (int u = 0; u < kVoxelPerThread; ++u) {
    const int i = tile * kVoxelTile + warp * (32 * kVoxelPerThread) + u * 32 + lane;
    code[u] = i < s.n ? __ldcg(keys + i) : 0;
    idx[u] = i < s.n ? __ldcg(index + i) : 0xffffffffu;                  // no point has this index (n <= kVoxelMaxTiles * kVoxelTile)
  }
  // digit counts of all tiles: a thread adds up four digits over every eighth tile
  {
    const int d4 = threadIdx.x & 63, part = threadIdx.x >> 6;
    const uint4* hist = reinterpret_cast<const uint4*>(s.hist + static_cast<size_t>(pass) * s.tiles * 256) + d4;
    uint4 total = make_uint4(0, 0, 0, 0), before = total;
#pragma unroll 8
    for (int t = part; t < s.tiles; t += kVoxelThreads / 64) {
      const uint4 c = __ldcg(hist + t * 64);
      const uint32_t e = t < tile ? 0xffffffffu : 0u;
      total.x += c.x; total.y += c.y; total.z += c.z; total.w += c.w;
      before.x += c.x & e; before.y += c.y & e; before.z += c.z & e; before.w += c.w & e;
    }
    if (threadIdx.x < 256) s_total[threadIdx.x] = s_before[threadIdx.x] = 0;
    for (int k = lane; k < 256; k += 32) s_warp[warp][k] = 0;
    __syncthreads();
    atomicAdd(&s_total[4 * d4], total.x); atomicAdd(&s_total[4 * d4 + 1], total.y);
    atomicAdd(&s_total[4 * d4 + 2], total.z); atomicAdd(&s_total[4 * d4 + 3], total.w);
    atomicAdd(&s_before[4 * d4], before.x); atomicAdd(&s_before[4 * d4 + 1], before.y);
    atomicAdd(&s_before[4 * d4 + 2], before.z); atomicAdd(&s_before[4 * d4 + 3], before.w);
  }
#pragma unroll
  for (int u = 0; u < kVoxelPerThread; ++u) {
    const bool real = idx[u] != 0xffffffffu;
    const uint32_t digit = static_cast<uint32_t>(voxel_key(code[u], axis_bits) >> shift) & 255u;
    uint32_t peers = __ballot_sync(0xffffffffu, real);          // lanes with the same digit, bit by bit
    if (!real) peers = ~peers;
#pragma unroll
    for (int bit = 0; bit < 8; ++bit) {
      const bool one = (digit >> bit) & 1;
      const uint32_t same = __ballot_sync(0xffffffffu, one);
      peers &= one ? same : ~same;
    }
    const uint32_t lower = peers & ((1u << lane) - 1u);
    const uint32_t first = s_warp[warp][digit];
    rank[u] = first + __popc(lower);
    __syncwarp();
    if (real && lower == 0) s_warp[warp][digit] = first + __popc(peers);
    __syncwarp();
  }
  __syncthreads();
  if (threadIdx.x < 256) {
    const int d = threadIdx.x;
    // exclusive scans over the digits: of the totals of all tiles, and of this tile's own counts
    uint32_t own = 0;
#pragma unroll
    for (int w = 0; w < kVoxelWarps; ++w) own += s_warp[w][d];
    const uint32_t v = s_total[d];
    uint32_t incl = v, own_incl = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t up = __shfl_up_sync(0xffffffffu, incl, o), own_up = __shfl_up_sync(0xffffffffu, own_incl, o);
      if (lane >= o) {
        incl += up;
        own_incl += own_up;
      }
    }
    if (lane == 31) {
      s_scan[0][warp] = incl;
      s_scan[1][warp] = own_incl;
    }
    asm volatile("bar.sync 1, 256;" ::: "memory");
    uint32_t base = incl - v + s_before[d], local = own_incl - own;
#pragma unroll
    for (int w = 0; w < 8; ++w) {
      base += w < warp ? s_scan[0][w] : 0u;
      local += w < warp ? s_scan[1][w] : 0u;
    }
    s_global[d] = base - local;
#pragma unroll
    for (int w = 0; w < kVoxelWarps; ++w) {                     // local positions, over the warps of the tile
      const uint32_t c = s_warp[w][d];
      s_warp[w][d] = local;
      local += c;
    }
  }
  __syncthreads();
  // Through shared memory into the order of the digits: the stores are runs of consecutive words, and neighbouring lanes
  // mostly agree on destination tile and next digit, so that one atomic counts for all of them (points next to each other
  // share their high bits: an atomic each serialised on a handful of addresses).
#pragma unroll
  for (int u = 0; u < kVoxelPerThread; ++u) {
    if (idx[u] == 0xffffffffu) continue;
    const uint32_t digit = static_cast<uint32_t>(voxel_key(code[u], axis_bits) >> shift) & 255u;
    const uint32_t local = s_warp[warp][digit] + rank[u];
    s_code[local] = code[u];
    s_index[local] = idx[u];
  }
  __syncthreads();
  uint64_t* keys_out = s.keys(pass + 1);
  uint32_t* index_out = s.index(pass + 1);
  uint32_t* next = s.hist + static_cast<size_t>(pass + 1) * s.tiles * 256;
  const int count = min(kVoxelTile, s.n - tile * kVoxelTile);
#pragma unroll
  for (int u = 0; u < kVoxelPerThread; ++u) {
    const int local = u * kVoxelThreads + threadIdx.x;
    uint32_t cell = 0xffffffffu;                                // no such tile
    if (local < count) {
      const uint64_t c = s_code[local], key = voxel_key(c, axis_bits);
      const uint32_t pos = s_global[static_cast<uint32_t>(key >> shift) & 255u] + local;
      keys_out[pos] = c;
      index_out[pos] = s_index[local];
      cell = (pos / kVoxelTile) * 256 + (static_cast<uint32_t>(key >> (shift + 8)) & 255u);
    }
    if (pass + 1 < passes) {
      const uint32_t peers = __match_any_sync(0xffffffffu, cell);
      if (cell != 0xffffffffu && (peers & ((1u << lane) - 1u)) == 0) atomicAdd(next + cell, static_cast<uint32_t>(__popc(peers)));
    }
  }
}

__device__ __forceinline__ bool voxel_head(const uint64_t* keys, int i, int n) {
  return i < n && (i == 0 || __ldcg(keys + i) != __ldcg(keys + i - 1));
}

// All CTAs of the grid (launched cooperatively: they run at the same time) meet; `target` arrivals in total.  Gives up after about
// two seconds and returns false.
__device__ __forceinline__ bool voxel_barrier(const VoxelScratch& s, uint32_t target, VoxelShared& sh) {
  __syncthreads();
  if (threadIdx.x == 0) {
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(s.arrived) : "memory");
    const long long t0 = clock64();
    bool met = true;
    for (;;) {
      uint32_t now;
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(now) : "l"(s.arrived) : "memory");
      if (now >= target) break;
      if (clock64() - t0 > 4000000000LL) {
        met = false;
        break;
      }
    }
    sh.met = met;
  }
  __syncthreads();
  return sh.met;
}

// The sort in one cooperative launch: as many passes as the keys need, with a barrier over the grid behind each, then the number of
// first points of voxels per tile, for the gather and (`report`, in pinned host memory, kVoxelPending before; kVoxelFailed when a
// barrier gave up) for the host.  As a launch per pass, five whatever the extent, one to count and a wait for the stream, a frame of 196 k
// points took 67.9 us, this way 52.9 us; with extents of 3, 100, 1000 and 100,000 voxels (two, three, five and seven passes) 36, 52, 67 and
// 84 us where the launches took 49, 64, 78 and 113.
__global__ void __launch_bounds__(kVoxelThreads, 2) gct_voxel_sort_kernel(VoxelScratch s, volatile int32_t* report) {
  __shared__ VoxelShared sh;
  const int axis_bits = voxel_axis_bits(s), passes = voxel_passes(axis_bits);
  bool met = true;
  for (int pass = 0; pass < passes && met; ++pass) {
    for (int tile = blockIdx.x; tile < s.tiles; tile += gridDim.x) {
      voxel_pass(pass, passes, tile, axis_bits, s, sh);
      __syncthreads();
    }
    met = voxel_barrier(s, static_cast<uint32_t>(pass + 1) * gridDim.x, sh);
  }
  const uint64_t* keys = s.keys(passes);
  for (int tile = blockIdx.x; tile < s.tiles; tile += gridDim.x) {
    int count = 0;
#pragma unroll
    for (int u = 0; u < kVoxelPerThread; ++u)
      count += __syncthreads_count(met && voxel_head(keys, tile * kVoxelTile + u * kVoxelThreads + threadIdx.x, s.n));
    if (threadIdx.x == 0) {
      s.heads[tile] = count;
      report[tile] = met ? count : kVoxelFailed;
    }
  }
}

__global__ void __launch_bounds__(kVoxelThreads) gct_voxel_gather_kernel(const float* __restrict__ xyz, const float* __restrict__ rgb, float voxel_size,
                                                                         VoxelScratch s, float* __restrict__ centers, float* __restrict__ colors,
                                                                         int64_t* __restrict__ codes) {
  pdl_wait();
  __shared__ int s_base;
  __shared__ __align__(16) int s_count[kVoxelPerThread * kVoxelWarps];      // heads of (step, warp), in the order of the keys
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int passes = voxel_passes(voxel_axis_bits(s));
  const uint64_t* keys = s.keys(passes);
  const uint32_t* index = s.index(passes);
  if (warp == 0) {
    int before = 0;
    for (int t = lane; t < static_cast<int>(blockIdx.x); t += 32) before += s.heads[t];
    before = __reduce_add_sync(0xffffffffu, before);
    if (lane == 0) s_base = before;
  }
  bool head[kVoxelPerThread];
  uint32_t ballot[kVoxelPerThread], src[kVoxelPerThread];
#pragma unroll
  for (int u = 0; u < kVoxelPerThread; ++u) {
    const int i = blockIdx.x * kVoxelTile + u * kVoxelThreads + threadIdx.x;
    head[u] = voxel_head(keys, i, s.n);
    src[u] = i < s.n ? index[i] : 0u;
  }
#pragma unroll
  for (int u = 0; u < kVoxelPerThread; ++u) {
    ballot[u] = __ballot_sync(0xffffffffu, head[u]);
    if (lane == 0) s_count[u * kVoxelWarps + warp] = __popc(ballot[u]);
  }
  __syncthreads();
  // every warp scans the 64 counts: two per lane
  static_assert(kVoxelPerThread * kVoxelWarps == 64, "two counts per lane");
  const int c0 = s_count[2 * lane], c1 = s_count[2 * lane + 1];
  int incl = c0 + c1;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int up = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += up;
  }
  const int excl = incl - c0 - c1;
#pragma unroll
  for (int u = 0; u < kVoxelPerThread; ++u) {
    const int e = u * kVoxelWarps + warp;
    int at = s_base + __shfl_sync(0xffffffffu, (e & 1) ? excl + c0 : excl, e >> 1);
    if (!head[u]) continue;
    at += __popc(ballot[u] & ((1u << lane) - 1u));
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const int v = voxel_index(xyz[3 * src[u] + c], voxel_size);
      centers[3 * static_cast<int64_t>(at) + c] = __fmul_rn(__fadd_rn(static_cast<float>(v), 0.5f), voxel_size);
      colors[3 * static_cast<int64_t>(at) + c] = rgb[3 * src[u] + c];
    }
    codes[at] = static_cast<int64_t>(keys[blockIdx.x * kVoxelTile + u * kVoxelThreads + threadIdx.x]);
  }
}

// Scratch of a call: [keys 2][index 2][extent][hist][heads][arrived], 256-byte aligned parts.
VoxelScratch voxel_scratch(void* base, int64_t n, size_t* bytes) {
  VoxelScratch s = {};
  s.n = static_cast<int>(n);
  s.tiles = static_cast<int>((n + kVoxelTile - 1) / kVoxelTile);
  size_t off = 0;
  auto part = [&](size_t size) {
    const size_t at = off;
    off = (off + size + 255) & ~size_t(255);
    return static_cast<uint8_t*>(base) + at;
  };
  s.keys0 = reinterpret_cast<uint64_t*>(part(static_cast<size_t>(n) * 8));
  s.keys1 = reinterpret_cast<uint64_t*>(part(static_cast<size_t>(n) * 8));
  s.index0 = reinterpret_cast<uint32_t*>(part(static_cast<size_t>(n) * 4));
  s.index1 = reinterpret_cast<uint32_t*>(part(static_cast<size_t>(n) * 4));
  s.extent = reinterpret_cast<uint32_t*>(part(static_cast<size_t>(s.tiles) * 4));
  s.hist = reinterpret_cast<uint32_t*>(part(static_cast<size_t>(kVoxelMaxPasses) * s.tiles * 256 * 4));
  s.heads = reinterpret_cast<int32_t*>(part(static_cast<size_t>(s.tiles) * 4));
  s.arrived = reinterpret_cast<uint32_t*>(part(sizeof(uint32_t)));
  if (bytes != nullptr) *bytes = off;
  return s;
}

int grid_for(int64_t items) {
  const int64_t blocks = (items + 255) / 256;
  return static_cast<int>(blocks < 1 ? 1 : (blocks > 148 * 16 ? 148 * 16 : blocks));
}

}  // namespace

int frustum_cull(const float* pts, int64_t n, const float* R, const float* t, const int* device_strides, float fx, float fy, float cx,
                 float cy, int width, int height, float near_plane, float far_plane, uint8_t* visible, cudaStream_t stream) {
  if (pts == nullptr || visible == nullptr) return fail(GCT_ERR_INVALID, "gct_frustum_cull: null argument");
  if ((reinterpret_cast<uintptr_t>(pts) & 15) || (reinterpret_cast<uintptr_t>(visible) & 3))
    return fail(GCT_ERR_INVALID, "gct_frustum_cull: points must be 16-byte aligned, the mask 4-byte aligned");
  CullArgs a = {};
  if (device_strides != nullptr) {
    a.R_dev = R;
    a.t_dev = t;
    a.R_row = device_strides[0];
    a.R_col = device_strides[1];
    a.t_step = device_strides[2];
  } else {
    for (int i = 0; i < 9; ++i) a.R[i] = R[i];
    for (int i = 0; i < 3; ++i) a.t[i] = t[i];
  }
  a.fx = fx; a.fy = fy; a.cx = cx; a.cy = cy;
  a.near_plane = near_plane; a.far_plane = far_plane;
  a.W = width; a.H = height;
  auto axis = [](float c, int size, float* mid, float* in, float* out) {
    const float middle = 0.5f * (static_cast<float>(size) - 1.f), half = 0.5f * (static_cast<float>(size) + 1.f);
    const float margin = 1e-5f * (fabsf(c) + fabsf(static_cast<float>(size)) + 1.f);
    *mid = c - middle;
    *in = half - margin;
    *out = half + margin;
    if (size <= 0) *in = *out = -1.f;                      // no pixel: out wherever the projection is a number
  };
  axis(cx, width, &a.mid_u, &a.in_u, &a.out_u);
  axis(cy, height, &a.mid_v, &a.in_v, &a.out_v);
  a.depth_tame = near_plane > 1e-30f && far_plane < 1e30f;
  // The camera is read once per thread, so a thread takes many points: two waves at the most (64 registers, four CTAs per SM).
  GCT_CUDA_CHECK(launch_pdl(gct_frustum_cull_kernel, dim3(std::min(grid_for(n / 4), 148 * 8)), dim3(256), 0, stream, pts, a, visible, n));
  return GCT_OK;
}

static_assert(kVoxelMaxPoints == static_cast<int64_t>(kVoxelMaxTiles) * kVoxelTile, "limit of the sort");

int voxel_sort_layout(int64_t n, size_t* bytes, int* tiles) {
  if (n < 1 || n > kVoxelMaxPoints) return fail(GCT_ERR_INVALID, "voxel sort: number of points out of range");
  *tiles = voxel_scratch(nullptr, n, bytes).tiles;
  return GCT_OK;
}

int voxel_sort(const float* xyz, float voxel_size, int64_t n, void* scratch, int32_t* report, int64_t* voxels_out, cudaStream_t stream) {
  if (!(voxel_size > 0.f)) return fail(GCT_ERR_INVALID, "gct_voxel_morton: bad argument");
  const VoxelScratch s = voxel_scratch(scratch, n, nullptr);
  int sms = 148;
  const int rc = device_sm_count(&sms);
  if (rc != GCT_OK) return rc;
  unsigned flags = 0;
  GCT_CUDA_CHECK(cudaGetDeviceFlags(&flags));
  std::fill(report, report + s.tiles, kVoxelPending);
  GCT_CUDA_CHECK(launch_pdl(gct_voxel_code_kernel, dim3(s.tiles), dim3(kVoxelThreads), 0, stream, xyz, voxel_size, s));
  cudaLaunchConfig_t cfg = {};
  cfg.blockDim = dim3(kVoxelThreads);
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  // Two CTAs of the sort fit an SM: all tiles at once where there are 128 SMs.  The stream may own fewer than the device has (a green
  // context, a share of the device); the driver then refuses the launch, and half as many CTAs take twice as many tiles each.
  int grid = std::min(s.tiles, 2 * sms);
  for (;;) {
    cfg.gridDim = dim3(grid);
    const cudaError_t e = cudaLaunchKernelEx(&cfg, gct_voxel_sort_kernel, s, static_cast<volatile int32_t*>(report));
    if (e != cudaErrorCooperativeLaunchTooLarge || grid == 1) {
      GCT_CUDA_CHECK(e);
      break;
    }
    cudaGetLastError();                                // answered by the smaller launch
    grid /= 2;
  }
  // The counts are looked for where the kernel writes them: they are there some microseconds before the stream is seen to be idle.
  // Only for as long as the largest sort takes with nothing queued before it, and only in a program whose threads spin in waits anyway;
  // otherwise, and behind earlier work, the wait is the stream's, as the program chose it for the device.
  const volatile int32_t* counts = report;
  const unsigned schedule = flags & cudaDeviceScheduleMask;
  bool look = schedule == cudaDeviceScheduleAuto || schedule == cudaDeviceScheduleSpin;
  const auto until = std::chrono::steady_clock::now() + kVoxelLook;
  int64_t total = 0;
  for (int t = 0; t < s.tiles; ++t) {
    while (look && counts[t] == kVoxelPending) look = std::chrono::steady_clock::now() < until;
    if (counts[t] == kVoxelPending) {
      GCT_CUDA_CHECK(cudaStreamSynchronize(stream));
      if (counts[t] == kVoxelPending) return fail(GCT_ERR_DEVICE_STATUS, "voxelisation: the sort ended without a result");
    }
    if (counts[t] == kVoxelFailed) {
      GCT_CUDA_CHECK(cudaStreamSynchronize(stream));
      return fail(GCT_ERR_DEVICE_STATUS, "voxelisation: a barrier of the sort was not reached in time");
    }
    total += counts[t];
  }
  *voxels_out = total;
  return GCT_OK;
}

int voxel_gather(const float* xyz, const float* rgb, float voxel_size, int64_t n, void* scratch, float* centers, float* colors,
                 int64_t* codes, cudaStream_t stream) {
  const VoxelScratch s = voxel_scratch(scratch, n, nullptr);
  GCT_CUDA_CHECK(launch_pdl(gct_voxel_gather_kernel, dim3(s.tiles), dim3(kVoxelThreads), 0, stream, xyz, rgb, voxel_size, s, centers, colors, codes));
  return GCT_OK;
}
}  // namespace gct

extern "C" {

int gct_frustum_cull(const float* pts_dev, int64_t n, const float R_cw[9], const float t_cw[3], float fx, float fy, float cx,
                     float cy, int width, int height, float near_plane, float far_plane, uint8_t* visible_dev, void* stream) {
  using namespace gct;
  if (n < 0 || R_cw == nullptr || t_cw == nullptr) return fail(GCT_ERR_INVALID, "gct_frustum_cull: bad argument");
  if (n == 0) return GCT_OK;
  return frustum_cull(pts_dev, n, R_cw, t_cw, nullptr, fx, fy, cx, cy, width, height, near_plane, far_plane, visible_dev,
                      static_cast<cudaStream_t>(stream));
}

int gct_voxel_morton(const float* xyz_dev, const float* rgb_dev, float voxel_size, int64_t n, int64_t* codes_dev,
                     float* centers_dev, float* colors_dev, void* stream) {
  using namespace gct;
  if (n < 0 || !(voxel_size > 0.f)) return fail(GCT_ERR_INVALID, "gct_voxel_morton: bad argument");
  if (n == 0) return GCT_OK;
  if (xyz_dev == nullptr || rgb_dev == nullptr || codes_dev == nullptr || centers_dev == nullptr || colors_dev == nullptr)
    return fail(GCT_ERR_INVALID, "gct_voxel_morton: null argument");
  gct_voxel_morton_kernel<<<grid_for(n), 256, 0, static_cast<cudaStream_t>(stream)>>>(xyz_dev, rgb_dev, voxel_size, n, codes_dev,
                                                                                     centers_dev, colors_dev);
  GCT_CUDA_CHECK(cudaGetLastError());
  return GCT_OK;
}

int gct_mark_unique(const int64_t* sorted_dev, int64_t n, uint8_t* mask_dev, void* stream) {
  using namespace gct;
  if (n < 0) return fail(GCT_ERR_INVALID, "gct_mark_unique: bad argument");
  if (n == 0) return GCT_OK;
  if (sorted_dev == nullptr || mask_dev == nullptr) return fail(GCT_ERR_INVALID, "gct_mark_unique: null argument");
  gct_mark_unique_kernel<<<grid_for(n), 256, 0, static_cast<cudaStream_t>(stream)>>>(sorted_dev, n, mask_dev);
  GCT_CUDA_CHECK(cudaGetLastError());
  return GCT_OK;
}

}  // extern "C"

// pixlist.cu -- multi-pose pixel-list renderer with optical flow.
//
// Restates baseline/fm_render.py:151-224 (render_func_idx_quattrans and its _flow variant) and
// :130-144 (render_func_quat_cam) with the argument order of their render_func_rays calls fixed
// (they pass the Gaussians where the rays belong). Input rays are the reference's pixel_posei rows
// (x, y, c, pose): the camera ray is (x invF, y invF, c) of pose `pose` (poses: (n_poses, 7) =
// quaternion (4, scalar first), translation (3)); or render_func_quat_cam's pixel_list rows
// (x, y, c) of one pose, whose camera ray is ((x - 0.5) invF, (y - 0.5) aspect invF, c) -- the
// same model with focal lengths 1/invF and 1/(aspect invF) and the pixel offsets shifted.
// Outputs per ray: depth and alpha as render_func_rays computes them (culled at
// the renderer's density cut-off), optionally the softmax-weighted per-Gaussian features
// (fm_render's w applied to a feature table) and the dense weights w (N x rays), and the
// forward / backward optical flow to poses pose+1 / pose-1 (clamped), fm_render.py:186-222.
//
// Work:
//  * pixlist_prep_kernel builds, per (pose, Gaussian), the same float32 record and screen bound as
//    the image preprocess (fe_footprint.cuh) with focal lengths 1/invF, 1/(aspect invF) and the
//    principal point at 0 (pixel offsets (x - shift_x)/c, (y - shift_y)/c), and every pose's
//    rotation matrix;
//  * long lists are bucketed by pose and 16-pixel cell (count, bases, scatter; the order inside a
//    bucket is free, since a ray's result does not depend on its neighbours), so that a warp's
//    rays lie close together whatever the order of the list;
//  * pixlist_kernel gives a warp 64 rays, two per lane (fewer for short lists). Its lanes test 32
//    Gaussians at a time against the box around the warp's rays (one coalesced 16-byte load
//    each), queue the ones that reach it and evaluate them in pairs from shared memory with
//    packed f32x2 arithmetic, each ray still counting only the Gaussians whose own bound holds it,
//    in index order: results do not depend on how rays are grouped;
//  * with few Gaussians or few tests in all, or when the dense weights are wanted,
//    pixlist_direct_kernel tests every Gaussian for every ray.
// Testing every Gaussian for every ray bounded this path: 1.2 M rays of 16 poses (every other
// pixel of 640x480) and 1000 Gaussians took 782 us in image order and 4447 us shuffled; bucketed
// 192 and 218 us, 156 us of it pixlist_kernel, bound by the issue slots of its evaluations (99 M
// warp instructions, issue active 48%, 15 warps per SM at 120 registers; 80 registers for 24 warps
// spill and take 204 us, 32 rays per warp 237 us).
#include <algorithm>
#include <type_traits>

#include "fe_footprint.cuh"
#include "fe_kernels.cuh"

namespace fe {
namespace {

// Scratch of one call: pixel-offset bounds (ulo, uhi, vlo, vhi) of the k-sigma projection and
// record per (pose, Gaussian), rotation (9 floats in 12) per pose.
struct PixScratch {
  char* table;      // float4 bound and GaussRec per (pose, Gaussian)
  float* rot;
  uint32_t* count;  // bucket sizes, then their first slots; the cursor after the last bucket
  uint2* place;     // per ray of a slice: bucket and rank in it
  uint32_t* order;  // ray indices (within the slice) by bucket
};
constexpr int kRotStride = 12;

// The (pose, Gaussian) table: bounds and records in arrays of their own, which lets a warp read 32
// bounds in four lines, or interleaved, which gives the thread-per-ray kernel's scattered reads a
// hit's record beside its bound.
template <int BOUND, int RECORD>  // bytes from one to the next
struct PixTable {
  char *bnd, *rec;
  __device__ __forceinline__ float4& bound(int64_t i) const {
    return *reinterpret_cast<float4*>(bnd + i * BOUND);
  }
  __device__ __forceinline__ GaussRec& record(int64_t i) const {
    return *reinterpret_cast<GaussRec*>(rec + i * RECORD);
  }
  __device__ __forceinline__ PixTable from(int64_t i) const {
    return {bnd + i * BOUND, rec + i * RECORD};
  }
};
constexpr int kInterleaved = sizeof(float4) + sizeof(GaussRec);
using SplitTable = PixTable<sizeof(float4), sizeof(GaussRec)>;
using InterleavedTable = PixTable<kInterleaved, kInterleaved>;

// Scales the ray terms of a record whose |a0| is below 2^-50 or above 2^50 by the power of two that
// takes it to about one. z = psv / vsv and the density's |y|^2 / vsv do not change, and vsv = |a|^2
// stays clear of the ends of the float32 range, where the reciprocal of evaluate_pairs is not the
// division's. (Terms whose square or its reciprocal has no float32 are left: they give NaN, as the
// division does.)
__device__ __forceinline__ void normalise_record(GaussRec& g) {
  const float top = fmaxf(fmaxf(fabsf(g.a0[0]), fabsf(g.a0[1])), fabsf(g.a0[2]));
  if (!(top >= 0x1p-64f && top < 0x1p64f) || (top >= 0x1p-50f && top <= 0x1p50f)) return;
  const float s = __uint_as_float((254u - (__float_as_uint(top) >> 23)) << 23);
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    g.a0[c] *= s; g.a1[c] *= s; g.a2[c] *= s; g.b[c] *= s;
    g.y0[c] *= s; g.y1[c] *= s; g.y2[c] *= s;
  }
}

template <class Table>
__global__ void pixlist_prep_kernel(int n, int n_poses, const float* __restrict__ means,
                                    const float* __restrict__ prec,
                                    const float* __restrict__ logw,
                                    const float* __restrict__ poses, float fx, float fy,
                                    int cull_mode, float cull_param, Table tab,
                                    float* __restrict__ rot, uint32_t* __restrict__ count,
                                    int64_t n_count) {
  const int64_t total = (int64_t)n * n_poses;
  const float L = 4.f * fmaxf(fabsf(fx), fabsf(fy));  // expansion centres within four focal lengths
  const int64_t first = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int64_t step = (int64_t)gridDim.x * blockDim.x;
  for (int64_t k = first; k < n_count; k += step) count[k] = 0u;  // (the first slice's buckets)
  for (int64_t k = first; k < n_poses; k += step) {
    float R[9];
    quat_to_rot<float>(poses + 7 * k, R);
#pragma unroll
    for (int q = 0; q < 9; ++q) rot[kRotStride * k + q] = R[q];
  }
  for (int64_t idx = first; idx < total; idx += step) {
    const int k = (int)(idx / n);
    const int i = (int)(idx - (int64_t)k * n);
    float R[9];
    quat_to_rot<float>(poses + 7 * k, R);
    const CamTerms ct = camera_terms(means + 3 * (int64_t)i, prec + 9 * (int64_t)i, R,
                                     poses + 7 * k + 4);
    const float lw = logw[i];
    const float k2 = cutoff_k2(lw, cull_mode, cull_param);
    float4 b = make_float4(INFINITY, -INFINITY, INFINITY, -INFINITY);  // empty
    if (k2 > 0.f) {
      float ulo = 0.f, uhi = 0.f, vlo = 0.f, vhi = 0.f;
      if (screen_bounds(ct, k2, fx, fy, 0.f, 0.f, ulo, uhi, vlo, vhi) == kFootBounded) {
        const float margin = 0.02f;  // covers the float32 rounding of the bounds
        b = make_float4(ulo - margin, uhi + margin, vlo - margin, vhi + margin);
      } else {
        b = make_float4(-INFINITY, INFINITY, -INFINITY, INFINITY);
      }
    }
    tab.bound(idx) = b;
    GaussRec g;
    make_record(ct, lw, fx, fy, 0.f, 0.f, 0.f, 0.f, -L, L, -L, L, g);
    if (std::is_same<Table, SplitTable>::value) normalise_record(g);
    tab.record(idx) = g;
  }
}

// Camera-frame point of pose `a` at ray parameter z, seen from pose `b`: pixel offsets (x, y).
__device__ __forceinline__ void reproject(const float* poses, const float* rot, int a, int b,
                                          float rx, float ry, float rz, float z, float inv_f,
                                          float& x, float& y) {
  const float* Ra = rot + (int64_t)kRotStride * a;
  const float* Rb = rot + (int64_t)kRotStride * b;
  const float* ta = poses + 7 * (int64_t)a + 4;
  const float* tb = poses + 7 * (int64_t)b + 4;
  // world = (ray z) @ Ra + ta;  pt = (world - tb) @ Rb^T
  const float cx = rx * z, cy = ry * z, cz = rz * z;
  float w[3];
  for (int j = 0; j < 3; ++j) w[j] = cx * Ra[0 * 3 + j] + cy * Ra[1 * 3 + j] + cz * Ra[2 * 3 + j] + ta[j];
  float p[3];
  for (int j = 0; j < 3; ++j)
    p[j] = (w[0] - tb[0]) * Rb[j * 3 + 0] + (w[1] - tb[1]) * Rb[j * 3 + 1] + (w[2] - tb[2]) * Rb[j * 3 + 2];
  x = p[0] / (p[2] * inv_f);
  y = p[1] / (p[2] * inv_f);
}

// A ray on the unit-depth plane. The record is evaluated on the ray (u/fx, v/fy, 1) with pixel
// offsets u = (x - shift_x)/c, v = (y - shift_y)/c; the parameter of the input ray
// ((x - shift_x) inv_f, (y - shift_y) aspect inv_f, c), which the softmax logits, the z > 0 mask
// and the depth use, is z / c.
struct PixRay {
  float x, y, c, ic, u, v;
  int k;
};

__device__ __forceinline__ PixRay load_ray(const float* __restrict__ rays, int64_t j,
                                           const PixRayModel& rm, int n_poses) {
  const float* row = rays + rm.stride * j;
  PixRay r;
  r.x = row[0]; r.y = row[1]; r.c = row[2];
  r.k = 0;
  if (rm.stride == 4) {
    r.k = (int)row[3];  // astype(int); out-of-range indices clamp, as JAX gathers do
    r.k = min(max(r.k, 0), n_poses - 1);
  }
  r.ic = 1.f / r.c;
  r.u = (r.x - rm.shift_x) * r.ic;
  r.v = (r.y - rm.shift_y) * r.ic;
  return r;
}

__device__ __forceinline__ bool in_bound(const float4& b, float u, float v) {
  return u >= b.x && u <= b.y && v >= b.z && v <= b.w;
}

// ---- bucketing ----------------------------------------------------------------------------------
// Bucket of a ray: pose (low bits) x Morton code of its 16-pixel cell, wrapped at 64 cells each
// way. Neighbouring buckets of a pose are neighbouring cells; rays that share a bucket only by
// wrapping, or buckets shared by poses 2^pose_bits apart, cost time in pixlist_kernel, not results.
constexpr int kCellBits = 6;  // cells per axis of a pose: 64 x 16 pixels
constexpr float kCellInv = 1.f / 16.f;
constexpr int kMaxPoseBits = 6;
constexpr int kBucketThreads = 256;
constexpr int kBucketPer = 16;  // buckets per thread of the bases kernel
// Rays per slice: bounds the order's scratch (12 B per ray).
constexpr int64_t kSliceRays = INT64_C(1) << 22;

__device__ __forceinline__ uint32_t spread_bits(uint32_t x) {  // bit i of x (6 bits) to bit 2 i
  x = (x | (x << 4)) & 0x30fu;
  x = (x | (x << 2)) & 0x333u;
  return (x | (x << 1)) & 0x555u;
}

__device__ __forceinline__ uint32_t ray_bucket(const PixRay& r, int pose_bits) {
  // (saturating conversions: non-finite offsets land in some cell)
  const uint32_t mask = (1u << kCellBits) - 1u;
  const uint32_t cu = (uint32_t)__float2int_rd(r.u * kCellInv) & mask;
  const uint32_t cv = (uint32_t)__float2int_rd(r.v * kCellInv) & mask;
  const uint32_t pose = (uint32_t)r.k & ((1u << pose_bits) - 1u);
  return (pose << (2 * kCellBits)) | spread_bits(cu) | (spread_bits(cv) << 1);
}

// Bucket and rank of every ray; lanes of one bucket share one atomic.
__global__ void __launch_bounds__(kBucketThreads) pixlist_count_kernel(
    int64_t n_rays, const float* __restrict__ rays, PixRayModel rm, int n_poses, int pose_bits,
    uint32_t* __restrict__ count, uint2* __restrict__ place) {
  const int lane = threadIdx.x & 31;
  const int64_t j = blockIdx.x * (int64_t)kBucketThreads + threadIdx.x;
  const bool valid = j < n_rays;
  uint32_t b = 0xffffffffu;
  if (valid) b = ray_bucket(load_ray(rays, j, rm, n_poses), pose_bits);
  const uint32_t same = __match_any_sync(0xffffffffu, b);
  const int leader = __ffs(same) - 1;
  uint32_t base = 0;
  if (valid && lane == leader) base = atomicAdd(&count[b], (uint32_t)__popc(same));
  base = __shfl_sync(0xffffffffu, base, leader);
  if (valid) place[j] = make_uint2(b, base + (uint32_t)__popc(same & ((1u << lane) - 1u)));
}

// First slot of every bucket, in place of its size: a block takes kBucketThreads * kBucketPer
// consecutive buckets and one range of slots for all of them (the blocks' order is free).
__global__ void __launch_bounds__(kBucketThreads) pixlist_bases_kernel(
    uint32_t* __restrict__ count, uint32_t* __restrict__ cursor) {
  __shared__ uint32_t ws[kBucketThreads / 32];
  __shared__ uint32_t block_base;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint4* mine = reinterpret_cast<uint4*>(count) +
                (blockIdx.x * (int64_t)kBucketThreads + threadIdx.x) * (kBucketPer / 4);
  uint4 c[kBucketPer / 4];
  uint32_t sum = 0;
#pragma unroll
  for (int q = 0; q < kBucketPer / 4; ++q) {
    c[q] = mine[q];
    sum += c[q].x + c[q].y + c[q].z + c[q].w;
  }
  uint32_t incl = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  if (lane == 31) ws[warp] = incl;
  __syncthreads();
  uint32_t before = 0, total = 0;
#pragma unroll
  for (int w = 0; w < kBucketThreads / 32; ++w) {
    if (w < warp) before += ws[w];
    total += ws[w];
  }
  if (threadIdx.x == 0) block_base = total ? atomicAdd(cursor, total) : 0u;
  __syncthreads();
  uint32_t at = block_base + before + incl - sum;
#pragma unroll
  for (int q = 0; q < kBucketPer / 4; ++q) {
    uint4 o;
    o.x = at; at += c[q].x;
    o.y = at; at += c[q].y;
    o.z = at; at += c[q].z;
    o.w = at; at += c[q].w;
    mine[q] = o;
  }
}

__global__ void __launch_bounds__(kBucketThreads) pixlist_scatter_kernel(
    int64_t n_rays, const uint32_t* __restrict__ base, const uint2* __restrict__ place,
    uint32_t* __restrict__ order) {
  const int64_t j = blockIdx.x * (int64_t)kBucketThreads + threadIdx.x;
  if (j >= n_rays) return;
  const uint2 p = place[j];
  order[base[p.x] + p.y] = (uint32_t)j;
}

// ---- rendering ----------------------------------------------------------------------------------

constexpr int kPixWarps = 4;
constexpr int kMaxF = 16;
// Two queued Gaussians, field by field: 24 record fields and 4 bounds as pairs; 60 words keep the
// 16-byte loads aligned and the building stores at two-way bank conflicts.
constexpr int kPairFields = 28;
constexpr int kPairWords = 60;

// Peak of one record along the ray at offsets (u, v): z of the input ray and log2 density.
__device__ __forceinline__ void eval_record(const GaussRec& g, float u, float v, float ic,
                                            float& z, float& s2) {
  const float du = u - g.uc, dv = v - g.vc;
  float a[3], y[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    a[c] = fmaf(g.a2[c], dv, fmaf(g.a1[c], du, g.a0[c]));
    y[c] = fmaf(g.y2[c], dv, fmaf(g.y1[c], du, g.y0[c]));
  }
  const float vsv = fmaf(a[2], a[2], fmaf(a[1], a[1], a[0] * a[0]));
  const float psv = fmaf(a[2], g.b[2], fmaf(a[1], g.b[1], a[0] * g.b[0]));
  const float yy = fmaf(y[2], y[2], fmaf(y[1], y[1], y[0] * y[0]));
  const float qi = 1.f / vsv;
  z = psv * qi * ic;
  s2 = fmaf(-0.5f * kLog2e * yy, qi, g.c2);
}

// The call's outputs (NULL: not wanted) and what the optional ones need.
struct PixOut {
  float *depth, *alpha, *flow_next, *flow_prev, *feats, *weights;
  int64_t weight_stride;
  int nf, n_poses;
  const float *poses, *rot;
  float beta3, nb2;
};

// Outputs of ray j from its sums; tab is its pose's.
template <bool FEAT, class Table>
__device__ __forceinline__ void write_ray(const PixOut& o, int64_t j, const PixRay& r, int n,
                                          const Table& tab, float inv_f,
                                          float A, float m, float W, float Z,
                                          const float (&F)[FEAT ? kMaxF : 1]) {
  const float iw = W > 0.f ? 1.f / W : 0.f;
  const float zd = Z * iw;  // parameter of the ray (x inv_f, y inv_f, c)
  o.depth[j] = zd;
  o.alpha[j] = -expm1f(-A);
  if (FEAT && o.feats) {
#pragma unroll
    for (int f = 0; f < (FEAT ? kMaxF : 1); ++f)
      if (f < o.nf) o.feats[j * o.nf + f] = F[f] * iw;
  }
  if (o.weights) {  // dense softmax weights (rows: Gaussians), a second pass over the Gaussians
    for (int i = 0; i < n; ++i) {
      float wi = 0.f;
      if (W > 0.f && in_bound(tab.bound(i), r.u, r.v)) {
        float z, s2;
        eval_record(tab.record(i), r.u, r.v, r.ic, z, s2);
        if (z > 0.f) wi = ex2_approx(fmaf(o.beta3, s2, o.nb2 * z) - m) * iw;
      }
      o.weights[(int64_t)i * o.weight_stride + j] = wi;
    }
  }
  const float rxf = r.x * inv_f, ryf = r.y * inv_f;
  float x, y;
  if (o.flow_next) {
    reproject(o.poses, o.rot, r.k, min(r.k + 1, o.n_poses - 1), rxf, ryf, r.c, zd, inv_f, x, y);
    o.flow_next[2 * j] = -(x - r.x);
    o.flow_next[2 * j + 1] = -(y - r.y);
  }
  if (o.flow_prev) {
    reproject(o.poses, o.rot, r.k, max(r.k - 1, 0), rxf, ryf, r.c, zd, inv_f, x, y);
    o.flow_prev[2 * j] = -(x - r.x);
    o.flow_prev[2 * j + 1] = -(y - r.y);
  }
}

// Few Gaussians, or dense weights wanted (a write per ray and Gaussian, along the list, outweighs
// the tests): a thread per ray in the order given, every Gaussian's bound tested by every ray
// (loaded eight at a time), the ones that hold it evaluated in index order.
template <bool FEAT>
__global__ void __launch_bounds__(128) pixlist_direct_kernel(
    int n, InterleavedTable tab, int64_t n_rays, const float* __restrict__ rays, PixRayModel rm,
    const float* __restrict__ feats, PixOut o) {
  for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < n_rays;
       j += (int64_t)gridDim.x * blockDim.x) {
    const PixRay r = load_ray(rays, j, rm, o.n_poses);
    const InterleavedTable pt = tab.from((int64_t)r.k * n);
    float A = 0.f, m = -1e30f, W = 0.f, Z = 0.f;
    float F[FEAT ? kMaxF : 1];
#pragma unroll
    for (int f = 0; f < (FEAT ? kMaxF : 1); ++f) F[f] = 0.f;
    auto eval = [&](int i) {
      float z, s2;
      eval_record(pt.record(i), r.u, r.v, r.ic, z, s2);
      A += ex2_approx(s2);
      if (z > 0.f) {
        const float l = fmaf(o.beta3, s2, o.nb2 * z);
        if (l > m) {
          const float sc = ex2_approx(m - l);
          W *= sc; Z *= sc;
#pragma unroll
          for (int f = 0; f < (FEAT ? kMaxF : 1); ++f) F[f] *= sc;
          m = l;
        }
        const float e = ex2_approx(l - m);
        W += e;
        Z = fmaf(e, z, Z);
        if (FEAT) {
#pragma unroll
          for (int f = 0; f < (FEAT ? kMaxF : 1); ++f)
            if (f < o.nf) F[f] = fmaf(e, feats[(int64_t)i * o.nf + f], F[f]);
        }
      }
    };
    constexpr int kBatch = 8;
    for (int i0 = 0; i0 < n; i0 += kBatch) {
      float4 b[kBatch];
#pragma unroll
      for (int t = 0; t < kBatch; ++t)
        b[t] = i0 + t < n ? pt.bound(i0 + t)
                          : make_float4(INFINITY, -INFINITY, INFINITY, -INFINITY);
      unsigned hit = 0;
#pragma unroll
      for (int t = 0; t < kBatch; ++t) hit |= in_bound(b[t], r.u, r.v) ? 1u << t : 0u;
      for (; hit; hit &= hit - 1) eval(i0 + __ffs(hit) - 1);
    }
    write_ray<FEAT>(o, j, r, n, pt, rm.inv_f, A, m, W, Z, F);
  }
}

__device__ __forceinline__ float warp_max(float x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x = fmaxf(x, __shfl_xor_sync(0xffffffffu, x, o));
  return x;
}

// Per-warp shared memory: the queue of Gaussians that reach the warp's rays, and the pairs of the
// batch under evaluation.
struct PixSmem {
  float pair[16][kPairWords];
  uint32_t queue[64];
};

// Build the pairs of the queue's first cnt (at most 32) Gaussians; an odd slot is in no bound.
__device__ __forceinline__ void build_pairs(PixSmem& sm, int lane, int cnt, const float4* bnd,
                                            const GaussRec* recs) {
  __syncwarp();
  if (lane < ((cnt + 1) & ~1)) {
    float f[kPairFields];
    if (lane < cnt) {
      const uint32_t i = sm.queue[lane];
      const float4* src = reinterpret_cast<const float4*>(recs + i);
#pragma unroll
      for (int q = 0; q < 6; ++q) {
        const float4 t = src[q];
        f[4 * q] = t.x; f[4 * q + 1] = t.y; f[4 * q + 2] = t.z; f[4 * q + 3] = t.w;
      }
      const float4 b = bnd[i];
      f[24] = b.x; f[25] = b.y; f[26] = b.z; f[27] = b.w;
    } else {
#pragma unroll
      for (int q = 0; q < kPairFields; ++q) f[q] = 0.f;
      f[24] = INFINITY; f[25] = -INFINITY;
    }
    float* dst = &sm.pair[lane >> 1][lane & 1];
#pragma unroll
    for (int q = 0; q < kPairFields; ++q) dst[2 * q] = f[q];
  }
  __syncwarp();
}

// The lane's rays (LR of them, in the halves of the packed sums) and their running sums.
template <int LR, bool FEAT>
struct LaneRays {
  float u[LR], v[LR], ic[LR];
  float m[2];
  f2_t A, W, Z;
  float F[LR][FEAT ? kMaxF : 1];
};

// The batch's Gaussians on the lane's rays. The two Gaussians of a pair are evaluated together
// with packed arithmetic and enter each ray's sums one after the other, so a ray's sums run over
// its Gaussians in index order whatever rays share the warp.
template <int LR, bool FEAT>
__device__ __forceinline__ void evaluate_pairs(const PixSmem& sm, int cnt, float beta3, float nb2,
                                               const float* feats, int nf, LaneRays<LR, FEAT>& t) {
  const f2_t B3 = f2_pack(beta3, beta3), NB2 = f2_pack(nb2, nb2);
  const f2_t KH = f2_pack(0.5f * kLog2e, 0.5f * kLog2e), ONE = f2_pack(1.f, 1.f);
  const int pairs = (cnt + 1) >> 1;
  for (int p = 0; p < pairs; ++p) {
    const ulonglong2* rp = reinterpret_cast<const ulonglong2*>(sm.pair[p]);
    // a0 a1 a2 b y0 y1 y2 (three fields each), uc, vc, c2, ulo, uhi, vlo, vhi
    const ulonglong2 r0 = rp[0], r1 = rp[1], r2 = rp[2], r3 = rp[3], r4 = rp[4], r5 = rp[5];
    const ulonglong2 r6 = rp[6], r7 = rp[7], r8 = rp[8], r9 = rp[9], r10 = rp[10], r11 = rp[11];
    const ulonglong2 r12 = rp[12], r13 = rp[13];
    float ulo[2], uhi[2], vlo[2], vhi[2];
    f2_unpack(r12.x, ulo[0], ulo[1]);
    f2_unpack(r12.y, uhi[0], uhi[1]);
    f2_unpack(r13.x, vlo[0], vlo[1]);
    f2_unpack(r13.y, vhi[0], vhi[1]);
    float s[2][2], l[2][2], z[2][2];  // [slot][ray]
#pragma unroll
    for (int q = 0; q < LR; ++q) {
      const f2_t du = sub2(f2_pack(t.u[q], t.u[q]), r10.y);
      const f2_t dv = sub2(f2_pack(t.v[q], t.v[q]), r11.x);
      const f2_t a0 = fma2(r3.x, dv, fma2(r1.y, du, r0.x));
      const f2_t a1 = fma2(r3.y, dv, fma2(r2.x, du, r0.y));
      const f2_t a2 = fma2(r4.x, dv, fma2(r2.y, du, r1.x));
      const f2_t y0 = fma2(r9.x, dv, fma2(r7.y, du, r6.x));
      const f2_t y1 = fma2(r9.y, dv, fma2(r8.x, du, r6.y));
      const f2_t y2 = fma2(r10.x, dv, fma2(r8.y, du, r7.x));
      const f2_t vsv = fma2(a2, a2, fma2(a1, a1, mul2(a0, a0)));
      const f2_t psv = fma2(a2, r5.y, fma2(a1, r5.x, mul2(a0, r4.y)));
      const f2_t yy = fma2(y2, y2, fma2(y1, y1, mul2(y0, y0)));
      float va, vb;
      f2_unpack(vsv, va, vb);
      // -1/vsv from the approximate reciprocal and a Newton step: the division's result, bit for
      // bit, for every vsv from 2^-126 up to 2^126 (all mantissas and exponents compared on GB300;
      // normalise_record keeps vsv well within). With the division here a list of 1.2 M rays takes
      // 242 us for 187.
      f2_t nqi = f2_pack(rcp_approx(-va), rcp_approx(-vb));
      nqi = fma2(nqi, fma2(vsv, nqi, ONE), nqi);
      const f2_t zz = mul2(mul2(psv, nqi), f2_pack(-t.ic[q], -t.ic[q]));
      const f2_t ss = fma2(mul2(KH, yy), nqi, r11.y);
      const f2_t ll = fma2(B3, ss, mul2(NB2, zz));
      f2_unpack(zz, z[0][q], z[1][q]);
      f2_unpack(ss, s[0][q], s[1][q]);
      f2_unpack(ll, l[0][q], l[1][q]);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        // (a ray outside the bound may not even be finite here)
        const bool in = t.u[q] >= ulo[h] && t.u[q] <= uhi[h] && t.v[q] >= vlo[h] && t.v[q] <= vhi[h];
        const bool front = in && z[h][q] > 0.f;
        s[h][q] = in ? s[h][q] : -INFINITY;
        z[h][q] = front ? z[h][q] : 0.f;
        l[h][q] = front ? l[h][q] : -INFINITY;
      }
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      if (LR == 1) { s[h][1] = -INFINITY; l[h][1] = -INFINITY; z[h][1] = 0.f; }
      t.A = add2(t.A, f2_pack(ex2_approx(s[h][0]), LR == 1 ? 0.f : ex2_approx(s[h][1])));
      if (l[h][0] > t.m[0] || (LR == 2 && l[h][1] > t.m[1])) {
        float sc[2] = {1.f, 1.f};
#pragma unroll
        for (int q = 0; q < LR; ++q) {
          if (l[h][q] > t.m[q]) {
            sc[q] = ex2_approx(t.m[q] - l[h][q]);
            t.m[q] = l[h][q];
          }
          if (FEAT) {
#pragma unroll
            for (int f = 0; f < (FEAT ? kMaxF : 1); ++f) t.F[q][f] *= sc[q];
          }
        }
        const f2_t S = f2_pack(sc[0], sc[1]);
        t.W = mul2(t.W, S);
        t.Z = mul2(t.Z, S);
      }
      const float e0 = ex2_approx(l[h][0] - t.m[0]);
      const float e1 = LR == 1 ? 0.f : ex2_approx(l[h][1] - t.m[1]);
      const f2_t E = f2_pack(e0, e1);
      t.W = add2(t.W, E);
      t.Z = fma2(E, f2_pack(z[h][0], z[h][1]), t.Z);
      if (FEAT && 2 * p + h < cnt) {
        const float* row = feats + (int64_t)sm.queue[2 * p + h] * nf;
#pragma unroll
        for (int q = 0; q < LR; ++q) {
          const float e = q ? e1 : e0;
          if (z[h][q] > 0.f) {  // (in front and within its bound)
#pragma unroll
            for (int f = 0; f < (FEAT ? kMaxF : 1); ++f)
              if (f < nf) t.F[q][f] = fmaf(e, row[f], t.F[q][f]);
          }
        }
      }
    }
  }
  __syncwarp();  // the pairs and the queue are rewritten next
}

// One warp per `wr` consecutive rays of the order (at most 32 LR; a power of two).
template <int LR, bool FEAT>
__global__ void __launch_bounds__(32 * kPixWarps) pixlist_kernel(
    int n, SplitTable tab, int64_t n_rays, int wr, const uint32_t* __restrict__ order,
    const float* __restrict__ rays, PixRayModel rm, const float* __restrict__ feats, PixOut o) {
  __shared__ __align__(16) PixSmem smem[kPixWarps];
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t first = (blockIdx.x * (int64_t)kPixWarps + warp) * wr;
  if (first >= n_rays) return;  // (uniform over the warp; no block barriers)
  const int64_t last = min(first + wr, n_rays);
  PixSmem& sm = smem[warp];
  const float kNone = __int_as_float(0x7fc00000);  // NaN: in no bound

  PixRay ray[LR];
  int64_t jj[LR];
  LaneRays<LR, FEAT> t;
  uint32_t todo[LR], any = 0;
  t.A = t.W = t.Z = 0;
  t.m[0] = t.m[1] = -1e30f;
#pragma unroll
  for (int q = 0; q < LR; ++q) {
    const int64_t at = first + 32 * q + lane;
    jj[q] = at < last ? (order ? (int64_t)order[at] : at) : -1;
    if (jj[q] >= 0) ray[q] = load_ray(rays, jj[q], rm, o.n_poses);
    else ray[q] = PixRay{0.f, 0.f, 1.f, 1.f, kNone, kNone, 0};
    t.ic[q] = ray[q].ic;
#pragma unroll
    for (int f = 0; f < (FEAT ? kMaxF : 1); ++f) t.F[q][f] = 0.f;
    todo[q] = __ballot_sync(full, jj[q] >= 0);
    any |= todo[q];
  }

  // The warp's rays pose by pose (mostly one).
  while (any) {
    int k = 0;
#pragma unroll
    for (int q = LR - 1; q >= 0; --q)
      if (todo[q]) k = __shfl_sync(full, ray[q].k, __ffs(todo[q]) - 1);
    float ulo = INFINITY, uhi = -INFINITY, vlo = INFINITY, vhi = -INFINITY;
    any = 0;
#pragma unroll
    for (int q = 0; q < LR; ++q) {
      const bool in = ray[q].k == k && ((todo[q] >> lane) & 1u);
      todo[q] &= ~__ballot_sync(full, in);
      any |= todo[q];
      t.u[q] = in ? ray[q].u : kNone;
      t.v[q] = in ? ray[q].v : kNone;
      // (a NaN offset lies in no bound, and fminf / fmaxf leave it out)
      ulo = fminf(ulo, t.u[q]); uhi = fmaxf(uhi, t.u[q]);
      vlo = fminf(vlo, t.v[q]); vhi = fmaxf(vhi, t.v[q]);
    }
    ulo = -warp_max(-ulo); uhi = warp_max(uhi);
    vlo = -warp_max(-vlo); vhi = warp_max(vhi);
    const float4* pb = &tab.bound((int64_t)k * n);
    const GaussRec* pr = &tab.record((int64_t)k * n);
    int qn = 0;  // queued Gaussians
    for (int c = 0; c < n; c += 128) {
      float4 b[4];
#pragma unroll
      for (int h = 0; h < 4; ++h) {
        const int i = c + 32 * h + lane;
        // (NaN reaches no box; an empty bound would reach one that rays with c = 0 make infinite)
        b[h] = i < n ? pb[i] : make_float4(kNone, kNone, kNone, kNone);
      }
#pragma unroll
      for (int h = 0; h < 4; ++h) {
        const bool hit = b[h].y >= ulo && b[h].x <= uhi && b[h].w >= vlo && b[h].z <= vhi;
        const uint32_t bal = __ballot_sync(full, hit);
        if (bal == 0u) continue;
        if (hit) sm.queue[qn + __popc(bal & ((1u << lane) - 1u))] = (uint32_t)(c + 32 * h + lane);
        qn += __popc(bal);
        if (qn >= 32) {
          build_pairs(sm, lane, 32, pb, pr);
          evaluate_pairs<LR, FEAT>(sm, 32, o.beta3, o.nb2, feats, o.nf, t);
          if (lane + 32 < qn) sm.queue[lane] = sm.queue[lane + 32];
          qn -= 32;
        }
      }
    }
    if (qn) {
      build_pairs(sm, lane, qn, pb, pr);
      evaluate_pairs<LR, FEAT>(sm, qn, o.beta3, o.nb2, feats, o.nf, t);
    }
  }

  float As[2], Ws[2], Zs[2];
  f2_unpack(t.A, As[0], As[1]);
  f2_unpack(t.W, Ws[0], Ws[1]);
  f2_unpack(t.Z, Zs[0], Zs[1]);

#pragma unroll
  for (int q = 0; q < LR; ++q)
    if (jj[q] >= 0)
      write_ray<FEAT>(o, jj[q], ray[q], n, tab.from((int64_t)ray[q].k * n), rm.inv_f, As[q], t.m[q],
                      Ws[q], Zs[q], t.F[q]);
}

inline size_t align256(size_t x) { return (x + 255) / 256 * 256; }

int pose_bits_for(int n_poses) {
  int b = 0;
  while (b < kMaxPoseBits && (1 << b) < n_poses) ++b;
  return b;
}

// Warps that fill the GPU.
constexpr int64_t kFillWarps = 152 * 16;
// Lists shorter than this are rendered in the order given: their warps hold a few rays each, and
// the bucketing launches would cost more than their wider boxes.
constexpr int64_t kOrderRays = 4 * kFillWarps;

// Few Gaussians, or a long list with few tests in all: every ray tests every Gaussian, since
// bucketing costs more than it saves. Per call, with flow, directly / bucketed: 1.2 M rays in image
// order, 20 Gaussians 56 / 75 us, 48 92 / 87, 100 154 / 106, 1000 782 / 192; 9 poses, in image
// order (shuffled), 112 K rays of 100 Gaussians 40 / 43 (44 / 43), 42 K of 300 45 / 52 (65 / 55),
// 112 K of 300 57 / 52 (105 / 57), 10 K of 1000 122 / 106 (164 / 105).
bool direct_list(int n, int64_t n_rays, bool weights) {
  if (n <= 40 || weights) return true;
  return n_rays >= kOrderRays && n <= 450 && n_rays <= INT64_C(16000000) / n;
}

// Rays per warp: 64 for long lists; short ones spread over the SMs, down to a ray per warp (which
// makes their order irrelevant).
int warp_rays(int64_t n_rays) {
  int wr = 64;
  while (wr > 1 && n_rays < (int64_t)wr * kFillWarps) wr >>= 1;
  return wr;
}

// Lays the scratch out from `base` (NULL to measure); `slice` rays are ordered at a time (0: none).
size_t carve(char* base, int n, int n_poses, int64_t slice, PixScratch& s) {
  size_t off = 0;
  auto take = [&](size_t bytes) {
    char* p = base ? base + off : nullptr;
    off += align256(bytes);
    return p;
  };
  const size_t total = (size_t)n * n_poses;
  s.table = take((size_t)kInterleaved * total);
  s.rot = reinterpret_cast<float*>(take(sizeof(float) * kRotStride * (size_t)n_poses));
  s.count = nullptr;
  s.place = nullptr;
  s.order = nullptr;
  if (slice > 0) {
    const size_t buckets = (size_t)1 << (2 * kCellBits + pose_bits_for(n_poses));
    s.count = reinterpret_cast<uint32_t*>(take(sizeof(uint32_t) * (buckets + 1)));
    s.place = reinterpret_cast<uint2*>(take(sizeof(uint2) * (size_t)slice));
    s.order = reinterpret_cast<uint32_t*>(take(sizeof(uint32_t) * (size_t)slice));
  }
  return off;
}

}  // namespace

size_t pixlist_scratch_bytes(int n, int n_poses, int64_t ordered_rays) {
  PixScratch s;
  return carve(nullptr, n, n_poses, std::min(ordered_rays, kSliceRays), s);
}

int64_t pixlist_ordered_rays(int n, int64_t n_rays, bool weights) {
  return n_rays >= kOrderRays && !direct_list(n, n_rays, weights) ? n_rays : 0;
}

void launch_render_pixels(int n, int n_poses, const float* means, const float* prec,
                          const float* logw, const float* poses, int64_t n_rays, const float* rays,
                          const PixRayModel& rm, float beta2, float beta3, int cull_mode,
                          float cull_param, const float* feats, int nf, float* depth, float* alpha,
                          float* flow_next, float* flow_prev, float* out_feats, float* weights,
                          int64_t ordered_rays, void* scratch, cudaStream_t st) {
  if (n_rays <= 0) return;
  const int64_t slice = std::min(n_rays, ordered_rays > 0 ? kSliceRays : n_rays);
  PixScratch s;
  carve(static_cast<char*>(scratch), n, n_poses, ordered_rays > 0 ? slice : 0, s);
  const bool direct = direct_list(n, n_rays, weights != nullptr);
  const int bits = pose_bits_for(n_poses);
  const int64_t buckets = INT64_C(1) << (2 * kCellBits + bits);
  const InterleavedTable mixed{s.table, s.table + sizeof(float4)};
  const SplitTable split{s.table, s.table + sizeof(float4) * (size_t)n * n_poses};
  {
    const int64_t b = (std::max<int64_t>((int64_t)n * n_poses, n_poses) + 127) / 128;
    const unsigned grid = (unsigned)std::min<int64_t>(b, 152 * 16);
    const float fx = 1.f / rm.inv_f, fy = 1.f / (rm.aspect * rm.inv_f);
    if (direct)
      pixlist_prep_kernel<<<grid, 128, 0, st>>>(n, n_poses, means, prec, logw, poses, fx, fy,
                                                cull_mode, cull_param, mixed, s.rot, nullptr, 0);
    else
      pixlist_prep_kernel<<<grid, 128, 0, st>>>(n, n_poses, means, prec, logw, poses, fx, fy,
                                                cull_mode, cull_param, split, s.rot, s.count,
                                                s.count ? buckets + 1 : 0);
  }
  for (int64_t r0 = 0; r0 < n_rays; r0 += slice) {
    const int64_t m = std::min(slice, n_rays - r0);
    const float* rows = rays + rm.stride * r0;
    if (ordered_rays > 0) {
      const unsigned grid = (unsigned)((m + kBucketThreads - 1) / kBucketThreads);
      if (r0 > 0) cudaMemsetAsync(s.count, 0, sizeof(uint32_t) * (size_t)(buckets + 1), st);
      pixlist_count_kernel<<<grid, kBucketThreads, 0, st>>>(m, rows, rm, n_poses, bits, s.count,
                                                            s.place);
      pixlist_bases_kernel<<<(unsigned)(buckets / (kBucketThreads * kBucketPer)), kBucketThreads, 0,
                             st>>>(s.count, s.count + buckets);
      pixlist_scatter_kernel<<<grid, kBucketThreads, 0, st>>>(m, s.count, s.place, s.order);
    }
    auto at = [&](float* p, int64_t width) { return p ? p + width * r0 : nullptr; };
    const PixOut o{depth + r0, alpha + r0, at(flow_next, 2), at(flow_prev, 2), at(out_feats, nf),
                   at(weights, 1), n_rays, nf, n_poses, poses, s.rot,
                   beta3, -beta2 * kLog2e};
    if (direct) {
      const unsigned grid = (unsigned)std::min<int64_t>((m + 127) / 128, 152 * 32);
      if (feats)
        pixlist_direct_kernel<true><<<grid, 128, 0, st>>>(n, mixed, m, rows, rm, feats, o);
      else
        pixlist_direct_kernel<false><<<grid, 128, 0, st>>>(n, mixed, m, rows, rm, feats, o);
      continue;
    }
    const int wr = warp_rays(m);
    const int64_t per_block = (int64_t)kPixWarps * wr;
    const unsigned grid = (unsigned)((m + per_block - 1) / per_block);
    auto go = [&](auto kern) {
      kern<<<grid, 32 * kPixWarps, 0, st>>>(n, split, m, wr, s.order, rows, rm, feats, o);
    };
    if (wr > 32) {
      if (feats) go(pixlist_kernel<2, true>); else go(pixlist_kernel<2, false>);
    } else {
      if (feats) go(pixlist_kernel<1, true>); else go(pixlist_kernel<1, false>);
    }
  }
}

}  // namespace fe

// loss.cu -- silhouette binary cross-entropy over the renders of a batch.
//
// The shape-from-silhouette loop of the reference (shape_from_silhouette.ipynb cell 12) scores a
// render's alpha against a target silhouette with
//     mean over pixels of -(t log a + (1 - t) log(1 - a)),  a clamped to [3e-8, 1 - 3e-8],
// and differentiates it with jax.grad. Here one kernel evaluates, for many renders laid out
// back to back in one pixel buffer (segment s = pixels [end[s-1], end[s])), every render's mean
// loss and the cotangent dL_s/dalpha of every pixel, which the blend backward consumes.
//
// float32 with the clamp applied to 1 - a rather than to a: 1 - a is exact for a >= 0.5
// (Sterbenz), so max(1 - a, 3e-8) equals 1 - min(a, 1 - 3e-8) evaluated exactly, whereas
// 1 - 3e-8 itself rounds to 1.0 in float32 (which would leave saturated pixels at log(0)).
// The per-render sums accumulate in float-float (two float32, about 48 bits) within a warp's run of
// pixels, and in float64 across warps: GB300 computes and converts float64 at a sixty-fourth of
// the float32 rate. With a float64 sum and product per pixel the kernel took 79 us on 16 renders of
// 640x480 (59 MB, 0.75 TB/s); it takes 18 us (3.3 TB/s), bound by instruction issue: a logarithm
// and a division per pixel, about 70 instructions in all.
#include <algorithm>

#include "fe_kernels.cuh"

namespace fe {
namespace {

constexpr float kClipAlpha = 3e-8f;
constexpr int kThreads = 256;
// Segment of pixel i: the first s with seg_end[s] > i.
__device__ __forceinline__ int segment_of(const int64_t* __restrict__ seg_end, int n_seg,
                                          int64_t i) {
  int lo = 0, hi = n_seg - 1;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (seg_end[mid] > i) hi = mid; else lo = mid + 1;
  }
  return lo;
}

// A float32 pair hi + lo (lo within half an ulp of hi): about 48 bits.
struct Pair {
  float hi, lo;
};

// x + y with the rounding of the float32 sum kept. A sum that is not finite has no error term.
__device__ __forceinline__ Pair add_pairs(Pair x, Pair y) {
  const float s = x.hi + y.hi, b = s - x.hi;
  const float e = (x.hi - (s - b)) + (y.hi - b) + (x.lo + y.lo);
  const float t = s + e;
  return fabsf(t) < INFINITY ? Pair{t, e - (t - s)} : Pair{s, 0.f};
}

// x times y.hi + y.lo.
__device__ __forceinline__ Pair scale(Pair x, Pair y) {
  const float p = x.hi * y.hi;
  const float e = fmaf(x.hi, y.hi, -p) + fmaf(x.hi, y.lo, x.lo * y.hi);
  return fabsf(p) < INFINITY ? Pair{p, e} : Pair{p, 0.f};
}

// 1 / pixels of render s (fewer than 2^48).
__device__ __forceinline__ Pair inv_count(const int64_t* __restrict__ seg_end, int s) {
  const int64_t n = seg_end[s] - (s > 0 ? seg_end[s - 1] : 0);
  const float nh = (float)n, nl = (float)(n - (int64_t)nh);
  const float r = 1.f / nh;
  return Pair{r, r * (fmaf(-r, nh, 1.f) - r * nl)};
}

// Loss of one pixel, and its derivative times `inv` to within one rounding. Targets of exactly 0
// or 1 (a silhouette) need one logarithm and one division: the other term's factor is 0 and its
// logarithm finite.
__device__ __forceinline__ float bce_pixel(float a, float t, Pair inv, float* g) {
  const float om = 1.f - a;
  const float ac = fmaxf(a, kClipAlpha);
  const float omc = fmaxf(om, kClipAlpha);
  const bool inside = (a > kClipAlpha) && (om > kClipAlpha);
  if ((t == 0.f || t == 1.f) && fabsf(a) < INFINITY) {
    const float x = t == 1.f ? ac : omc;
    const float d = inside ? (t == 1.f ? -1.f : 1.f) / x : 0.f;
    const float p = d * inv.hi;
    *g = p + fmaf(d, inv.lo, fmaf(d, inv.hi, -p));
    return -logf(x);
  }
  const Pair p = scale(Pair{inside ? (-t / ac + (1.f - t) / omc) : 0.f, 0.f}, inv);
  *g = p.hi + p.lo;
  return -(t * logf(ac) + (1.f - t) * logf(omc));
}

// A warp takes a contiguous run of pixels and goes through it render by render, four pixels per
// lane and step (16-byte accesses where all three buffers allow), keeping the render's sum in
// registers until the run leaves it.
__global__ void __launch_bounds__(kThreads) silhouette_bce_kernel(
    const float* __restrict__ alpha, const float* __restrict__ target,
    const int64_t* __restrict__ seg_end, int n_seg, int64_t n_pix, int64_t run, bool vec,
    float* __restrict__ galpha, double* __restrict__ loss) {
  const int lane = threadIdx.x & 31;
  const int64_t warp = ((int64_t)blockIdx.x * kThreads + threadIdx.x) >> 5;
  const int64_t end = min((warp + 1) * run, n_pix);
  for (int64_t at = warp * run; at < end;) {
    const int s = segment_of(seg_end, n_seg, at);
    const int64_t stop = s + 1 < n_seg ? min(seg_end[s], end) : end;
    const Pair inv = inv_count(seg_end, s);
    Pair sum{0.f, 0.f};
    auto add = [&](float x) {  // (the error terms' own sum needs no correction)
      const float t = sum.hi + x, b = t - sum.hi;
      sum.lo += (sum.hi - (t - b)) + (x - b);
      sum.hi = t;
    };
#pragma unroll 2
    for (int64_t u = (at >> 2) + lane; u < (stop + 3) >> 2; u += 32) {
      const int64_t i = 4 * u;
      if (vec && i >= at && i + 4 <= stop) {
        const float4 a = *reinterpret_cast<const float4*>(alpha + i);
        const float4 t = *reinterpret_cast<const float4*>(target + i);
        float4 g;
        add(bce_pixel(a.x, t.x, inv, &g.x));
        add(bce_pixel(a.y, t.y, inv, &g.y));
        add(bce_pixel(a.z, t.z, inv, &g.z));
        add(bce_pixel(a.w, t.w, inv, &g.w));
        *reinterpret_cast<float4*>(galpha + i) = g;
      } else {
        for (int64_t j = max(i, at); j < min(i + 4, stop); ++j) {
          float g;
          add(bce_pixel(alpha[j], target[j], inv, &g));
          galpha[j] = g;
        }
      }
    }
    if (!(fabsf(sum.hi) < INFINITY)) sum.lo = 0.f;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
      sum = add_pairs(sum, Pair{__shfl_xor_sync(0xffffffffu, sum.hi, o),
                                __shfl_xor_sync(0xffffffffu, sum.lo, o)});
    if (lane == 0) {
      const Pair mean = scale(sum, inv);
      atomicAdd(&loss[s], (double)mean.hi + (double)mean.lo);
    }
    at = stop;
  }
}

}  // namespace

void launch_silhouette_bce(const float* alpha, const float* target, const int64_t* seg_end,
                           int n_seg, int64_t n_pix, float* galpha, double* loss,
                           cudaStream_t st) {
  if (n_pix <= 0 || n_seg <= 0) return;
  // Runs of whole 128-pixel steps: one step per warp until the warps fill the GPU once, then
  // longer runs (a second, partial wave of blocks took 24 us against 18 on 16 x 640x480).
  constexpr int64_t kStep = 128, kWarps = kThreads / 32;
  const int64_t fill = resident_ctas<silhouette_bce_kernel>(kThreads) * kWarps;
  const int64_t steps = (n_pix + kStep - 1) / kStep;
  const int64_t per = (steps + fill - 1) / fill;
  const int64_t warps = (steps + per - 1) / per;
  const bool vec = ((reinterpret_cast<uintptr_t>(alpha) | reinterpret_cast<uintptr_t>(target) |
                     reinterpret_cast<uintptr_t>(galpha)) & 15) == 0;
  silhouette_bce_kernel<<<(unsigned)((warps + kWarps - 1) / kWarps), kThreads, 0, st>>>(
      alpha, target, seg_end, n_seg, n_pix, per * kStep, vec, galpha, loss);
}

}  // namespace fe

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
// The per-render sums accumulate in float64 and the derivatives are the float64 quotients, rounded.
// GB300 computes and converts float64 at a sixty-fourth of the float32 rate: with a sum, a product
// and four conversions per pixel a call on 16 renders of 640x480 (59 MB) took 82 us. One addition
// is left of them; the conversion before it moves bits, and the quotient comes from float32
// products wherever those determine its rounding: 25.5 us. (Sums and quotients in two float32 took
// 23, with 48 bits.) Bound by instruction issue: a logarithm and a division per pixel, about 80
// instructions in all.
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

// Pixels of render s.
__device__ __forceinline__ int64_t pixels_of(const int64_t* __restrict__ seg_end, int s) {
  return seg_end[s] - (s > 0 ? seg_end[s - 1] : 0);
}

// 1 / n as two float32 (n below 2^48): hi rounded, lo the rest to within 2^-46 of hi.
struct Inverse {
  float hi, lo;
  int64_t n;
};
__device__ __forceinline__ Inverse inverse_of(int64_t n) {
  const float nh = (float)n, nl = (float)(n - (int64_t)nh);
  const float r = 1.f / nh;
  return Inverse{r, r * (fmaf(-r, nh, 1.f) - r * nl), n};
}

// (The float64 instructions stay out of line: inlined, the compiler issues them for every pixel and
// picks a result afterwards, 64 us for 26.)
__device__ __noinline__ float scaled_f64(float d, int64_t n) {
  return (float)((double)d * (1.0 / (double)n));
}

// d / n as float64 arithmetic rounds it to float32. The two float32 products are within 2^-45 of
// the exact quotient; where that leaves its rounding open (one pixel in 2^19, and anything that is
// not finite) the float64 product is formed.
__device__ __forceinline__ float scaled(float d, const Inverse& inv) {
  const float p = d * inv.hi;
  const float e = fmaf(d, inv.lo, fmaf(d, inv.hi, -p));
  const float m = fabsf(p) * 0x1p-44f;
  const float g = p + (e + m);
  if (g == p + (e - m)) return g;
  return scaled_f64(d, inv.n);
}

// Loss of one pixel, and its derivative over the render's pixels. Targets of exactly 0 or 1 (a
// silhouette) need one logarithm and one division: the other term's factor is 0 and its logarithm
// finite.
__device__ __forceinline__ float bce_pixel(float a, float t, const Inverse& inv, float* g) {
  const float om = 1.f - a;
  const float ac = fmaxf(a, kClipAlpha);
  const float omc = fmaxf(om, kClipAlpha);
  const bool inside = (a > kClipAlpha) && (om > kClipAlpha);
  if ((t == 0.f || t == 1.f) && fabsf(a) < INFINITY) {
    const float x = t == 1.f ? ac : omc;
    *g = scaled(inside ? (t == 1.f ? -1.f : 1.f) / x : 0.f, inv);
    return -logf(x);
  }
  *g = scaled(inside ? (-t / ac + (1.f - t) / omc) : 0.f, inv);
  return -(t * logf(ac) + (1.f - t) * logf(omc));
}

__device__ __noinline__ double widen_slow(float x) { return (double)x; }
// x as float64. By moving bits for what is neither zero, subnormal nor not finite: the conversion
// instruction runs at the float64 rate.
__device__ __forceinline__ double widen(float x) {
  const uint32_t b = __float_as_uint(x), mag = b & 0x7fffffffu;
  if (mag - 0x00800000u >= 0x7f000000u) return mag == 0u ? 0.0 : widen_slow(x);
  return __hiloint2double((int)((b & 0x80000000u) | ((mag >> 3) + 0x38000000u)), (int)(b << 29));
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
    const Inverse inv = inverse_of(pixels_of(seg_end, s));
    double sum = 0.0;
    auto add = [&](float x) { sum += widen(x); };
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
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (lane == 0) atomicAdd(&loss[s], sum * (1.0 / (double)inv.n));
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

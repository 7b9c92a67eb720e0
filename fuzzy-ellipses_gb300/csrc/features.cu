// features.cu -- softmax-weighted per-Gaussian features of an image render.
//
// fm_render returns the normalised softmax weights w (N, pixels) next to depth and alpha, "to
// compute color, DINO features, or any other per-Gaussian property" (baseline/fm_render.py:
// 104-109): feature(pixel) = sum_i w_i(pixel) f_i. On the tiled image path the weights never
// exist as a matrix: this pass runs after a forward render and reuses its per-pixel statistics
// (softmax maximum m and normaliser W, base 2), so w_i = 2^(l_i - m) / W for the tile's front
// Gaussians.
//
// One CTA per tile; a thread owns PX consecutive pixels of a row and up to FC features of each in
// registers. The tile's keys come kFeatChunk at a time: their records are expanded around the tile
// into pair-interleaved TilePairs in shared memory, with their FC features beside them. The
// weights of two records are evaluated together with the forward blend's packed arithmetic (so
// they sum to one against its normaliser), then each is spread over the features two at a time.
// Wider features take a pass over the keys per 32. One warp per tile, scalar weights and a pass
// per four features took 179 us for 16 features of a 637x479 view of 1000 Gaussians (0.26 T
// weights/s); this kernel takes 30 us (a whole call with 64 features of a 640x480 view 906 -> 220
// us), bound by the tiles with the most keys (1200 tiles on 152 SMs).
#include <algorithm>

#include "fe_kernels.cuh"
#include "fe_tilerec.cuh"

namespace fe {
namespace {

constexpr int kFeatChunk = 64;  // records per shared-memory stage

template <int FC>
struct FeatSmem {
  TilePair pair[kFeatChunk / 2];
  float4 feat[kFeatChunk][FC / 4];
  uint32_t gid[kFeatChunk];
};

// Weights (times W) of a record pair at the thread's pixels: 2^(l - m), with MASK 0 behind the
// camera and at pixels that take no weights (m infinite), whatever the logits are. The arithmetic
// of blend_group (blend_fwd.cu).
template <int PX, bool MASK>
__device__ __forceinline__ void pair_weights(const TilePair& p, const f2_t (&DU)[PX], f2_t DV,
                                             f2_t DVSQ, f2_t B3, f2_t NB2, const float (&m)[PX],
                                             float (&e0)[PX], float (&e1)[PX]) {
  const ulonglong2* rp = reinterpret_cast<const ulonglong2*>(&p);
  const ulonglong2 r0 = rp[0], r1 = rp[1], r2 = rp[2], r3 = rp[3], r4 = rp[4];
  const ulonglong2 r5 = rp[5], r6 = rp[6], r7 = rp[7], r8 = rp[8];
  const f2_t bv = fma2(r2.y, DVSQ, fma2(r1.x, DV, r0.x));
  const f2_t cv = fma2(r2.x, DV, r0.y);
  const f2_t bp = fma2(r4.x, DV, r3.x);
  const f2_t ev = sub2(DV, r8.y);
  const f2_t bn = fma2(mul2(r7.x, ev), ev, fma2(r5.y, ev, r4.y));
  const f2_t cn = fma2(r6.y, ev, r5.x);
#pragma unroll
  for (int k = 0; k < PX; ++k) {
    const f2_t vsv = fma2(fma2(r1.y, DU[k], cv), DU[k], bv);
    const f2_t psv = fma2(r3.y, DU[k], bp);
    const f2_t eu = sub2(DU[k], r8.x);
    const f2_t nq = fma2(fma2(r6.x, eu, cn), eu, bn);
    float va, vb;
    f2_unpack(vsv, va, vb);
    const f2_t qi = f2_pack(rcp_approx(va), rcp_approx(vb));
    const f2_t z = mul2(psv, qi);
    const f2_t s2 = fma2(nq, qi, r7.y);
    float l0, l1;
    f2_unpack(sub2(fma2(B3, s2, mul2(NB2, z)), f2_pack(m[k], m[k])), l0, l1);
    e0[k] = ex2_approx(l0);
    e1[k] = ex2_approx(l1);
    if (MASK) {
      float z0, z1;
      f2_unpack(z, z0, z1);
      e0[k] = z0 > 0.f && m[k] < INFINITY ? e0[k] : 0.f;
      e1[k] = z1 > 0.f && m[k] < INFINITY ? e1[k] : 0.f;
    }
  }
}

template <int TW, int TH, int PX, int FC>
__global__ void __launch_bounds__(TW * TH / PX) features_kernel(
    ViewsArg va, const uint64_t* __restrict__ keys, const uint2* __restrict__ ranges,
    const GaussRec* __restrict__ recs, const float* __restrict__ stats, int64_t stride, float nb2,
    float beta3, const float* __restrict__ feats, int nf, int per_pass, float* __restrict__ out) {
  constexpr int NT = TW * TH / PX, CW = TW / PX;
  __shared__ __align__(16) FeatSmem<FC> sm;
  chain_wait();
  const int tid = threadIdx.x;
  const uint32_t tile = blockIdx.x;
  const int vi = view_of_tile(va, tile);
  const ViewDev& V = view_at(va, vi);
  const int lt = (int)(tile - V.tile_base);
  const int tx = lt % V.gx, ty = lt / V.gx;
  const int ly = tid / CW, cx = tid % CW;
  const int v = ty * TH + ly, u0 = tx * TW + cx * PX;
  const GaussRec* vrec = recs + V.rec_base;
  const uint2 range = ranges[tile];
  const float hw = 0.5f * (TW - 1), hh = 0.5f * (TH - 1);
  const f2_t B3 = f2_pack(beta3, beta3), NB2 = f2_pack(nb2, nb2);
  const float dv = ly - hh;
  const f2_t DV = f2_pack(dv, dv), DVSQ = f2_pack(dv * dv, dv * dv);
  f2_t DU[PX];
  float m[PX], iw[PX];
  int64_t pix[PX];
  bool ok[PX];
  bool weights = true;  // every pixel of the warp takes some
#pragma unroll
  for (int k = 0; k < PX; ++k) {
    const float du = (cx * PX + k) - hw;
    DU[k] = f2_pack(du, du);
    ok[k] = v < V.H && u0 + k < V.W;
    pix[k] = V.pix_base + (int64_t)v * V.W + u0 + k;
    const float W = ok[k] ? stats[stride + pix[k]] : 0.f;
    // A pixel without front Gaussians has W = 0 and m at the forward's sentinel, one that an
    // infinite logit reaches W = NaN: no weights.
    iw[k] = W > 0.f ? 1.f / W : 0.f;
    m[k] = W > 0.f ? stats[pix[k]] : INFINITY;
    weights &= m[k] < INFINITY || !ok[k];
  }
  weights = __all_sync(0xffffffffu, weights);
  for (int c0 = 0; c0 < nf; c0 += per_pass) {
    const int cn = min(per_pass, nf - c0);  // at most FC
    f2_t acc[PX][FC / 2];
#pragma unroll
    for (int k = 0; k < PX; ++k)
#pragma unroll
      for (int j = 0; j < FC / 2; ++j) acc[k][j] = 0;
    for (uint32_t k0 = range.x; k0 < range.y; k0 += kFeatChunk) {
      const int nk = (int)min((uint32_t)kFeatChunk, range.y - k0);
      const int pairs = (nk + 1) >> 1;
      __syncthreads();  // the previous chunk is no longer read
      for (int r = tid; r < 2 * pairs; r += NT) {
        TileRec t;
        if (r < nk) {
          const uint32_t g_id = (uint32_t)keys[k0 + r];
          sm.gid[r] = g_id;
          const GaussRec g = vrec[g_id];
          tile_record(g, tx * TW + hw - g.uc, ty * TH + hh - g.vc, hw, hh, t);
        } else {
          null_tile_record(t);
        }
        const float* f = reinterpret_cast<const float*>(&t);
        float* dst = reinterpret_cast<float*>(&sm.pair[r >> 1]) + (r & 1);
#pragma unroll
        for (int i = 0; i < kRecFields; ++i) dst[2 * i] = f[i];
      }
      __syncthreads();
      float* sf = reinterpret_cast<float*>(sm.feat);
      for (int i = tid; i < 2 * pairs * FC; i += NT) {
        const int r = i / FC, j = i - r * FC;
        sf[i] = r < nk && j < cn ? feats[(int64_t)sm.gid[r] * nf + c0 + j] : 0.f;
      }
      __syncthreads();
      for (int p = 0; p < pairs; ++p) {
        const float2 front = sm.pair[p].f[18];
        float e0[PX], e1[PX];
        if (front.x != 0.f && front.y != 0.f && weights)
          pair_weights<PX, false>(sm.pair[p], DU, DV, DVSQ, B3, NB2, m, e0, e1);
        else
          pair_weights<PX, true>(sm.pair[p], DU, DV, DVSQ, B3, NB2, m, e0, e1);
        const ulonglong2* f0 = reinterpret_cast<const ulonglong2*>(sm.feat[2 * p]);
        const ulonglong2* f1 = reinterpret_cast<const ulonglong2*>(sm.feat[2 * p + 1]);
#pragma unroll
        for (int j = 0; j < FC / 4; ++j) {
          const ulonglong2 a = f0[j], b = f1[j];
#pragma unroll
          for (int k = 0; k < PX; ++k) {
            const f2_t E0 = f2_pack(e0[k], e0[k]), E1 = f2_pack(e1[k], e1[k]);
            acc[k][2 * j] = fma2(E1, b.x, fma2(E0, a.x, acc[k][2 * j]));
            acc[k][2 * j + 1] = fma2(E1, b.y, fma2(E0, a.y, acc[k][2 * j + 1]));
          }
        }
      }
    }
#pragma unroll
    for (int k = 0; k < PX; ++k) {
      if (!ok[k]) continue;
      float x[FC];
#pragma unroll
      for (int j = 0; j < FC / 2; ++j) {
        f2_unpack(acc[k][j], x[2 * j], x[2 * j + 1]);
        x[2 * j] *= iw[k];
        x[2 * j + 1] *= iw[k];
      }
      float* dst = out + pix[k] * nf + c0;
      const bool vec = (reinterpret_cast<uintptr_t>(dst) & 15) == 0;
#pragma unroll
      for (int j = 0; j < FC; j += 4) {
        if (vec && j + 4 <= cn) {
          *reinterpret_cast<float4*>(dst + j) = make_float4(x[j], x[j + 1], x[j + 2], x[j + 3]);
        } else {
#pragma unroll
          for (int q = 0; q < 4; ++q)
            if (j + q < cn) dst[j + q] = x[j + q];
        }
      }
    }
  }
}

template <int TW, int TH, int FC>
void launch_tiles(const ViewsArg& va, int64_t n_tiles, const uint64_t* keys, const uint2* ranges,
                  const GaussRec* recs, const float* stats, int64_t stride, float beta2,
                  float beta3, const float* feats, int nf, float* out, cudaStream_t st) {
  // Two pixels per thread: at four, few heavy tiles leave the GPU short of threads (a 301x300 view
  // of 4000 Gaussians: 1236 us against 1680), at one, large views repeat the record loads (308
  // against 347 us for 1280x720).
  constexpr int PX = 2;
  const int passes = (nf + FC - 1) / FC;
  launch_chained(va.chain, features_kernel<TW, TH, PX, FC>, (unsigned)n_tiles, TW * TH / PX, st,
                 va, keys, ranges, recs, stats, stride, -beta2 * kLog2e, beta3, feats, nf,
                 (nf + passes - 1) / passes, out);
}

template <int TW, int TH>
void launch_width(const ViewsArg& va, int64_t n_tiles, const uint64_t* keys, const uint2* ranges,
                  const GaussRec* recs, const float* stats, int64_t stride, float beta2,
                  float beta3, const float* feats, int nf, float* out, cudaStream_t st) {
  auto go = [&](auto launch) {
    launch(va, n_tiles, keys, ranges, recs, stats, stride, beta2, beta3, feats, nf, out, st);
  };
  if (nf <= 4) go(launch_tiles<TW, TH, 4>);
  else if (nf <= 8) go(launch_tiles<TW, TH, 8>);
  else if (nf <= 16) go(launch_tiles<TW, TH, 16>);
  else go(launch_tiles<TW, TH, 32>);
}

}  // namespace

void launch_features(const ViewsArg& va, int tile_w, int tile_h, int64_t n_tiles,
                     const uint64_t* keys, const uint2* ranges, const GaussRec* recs,
                     const float* stats, int64_t stats_stride, float beta2, float beta3,
                     const float* feats, int nf, float* out, cudaStream_t st) {
  if (n_tiles <= 0 || nf <= 0) return;
  if (tile_w == 8 && tile_h == 8)
    launch_width<8, 8>(va, n_tiles, keys, ranges, recs, stats, stats_stride, beta2, beta3, feats,
                       nf, out, st);
  else if (tile_w == 32 && tile_h == 8)
    launch_width<32, 8>(va, n_tiles, keys, ranges, recs, stats, stats_stride, beta2, beta3,
                        feats, nf, out, st);
  else
    launch_width<16, 16>(va, n_tiles, keys, ranges, recs, stats, stats_stride, beta2, beta3,
                         feats, nf, out, st);
}

}  // namespace fe

// blend_fwd.cu -- per-tile forward blend: depth softmax and alpha in one pass.
//
// Persistent CTAs take screen tiles from a device-side work counter (one launch covers any number
// of uneven renders); each thread owns PX pixels of one tile row. A tile's keys are taken in
// chunks of 2 CH: the chunk's Gaussian records (96 B each) are staged in shared memory by 1-D TMA
// bulk copies (cp.async.bulk, one per record, completing on an mbarrier; every wait bounded)
// while the previous chunk is evaluated, then each thread re-expands its records around
// the tile centre into pair-interleaved TilePairs (two records per 160 B, field by field) in a
// double-buffered shared-memory ring; the Gaussian ids of the chunk after are read one chunk
// ahead of that. No record stream is written to or read from HBM for the forward. Two records
// are evaluated together with packed
// f32x2 arithmetic, so each 16-byte shared load yields two ready operands and every polynomial,
// logit and accumulation step is one instruction for two evaluations. Per (pixel, Gaussian):
//     vsv = V(du,dv)   psv = P(du,dv)   nq = N(du-cu, dv-cv)    (row-constant parts shared by
//                                                                the thread's PX pixels)
//     q = rcp(vsv); z = psv q; s2 = C + nq q                    (z: peak ray parameter,
//                                                                s2: log2 peak density)
//     A += 2^s2                                                 (alpha, all Gaussians)
//     l = beta3 s2 - beta2 log2(e) z, masked to z > 0            (log2 softmax logit; the mask is
//                                                                skipped for pairs whose psv is
//                                                                positive over the whole tile)
// and an online max (updated once per group of records) keeps the softmax in one pass:
//     W = sum 2^(l-m), Z = sum 2^(l-m) z, depth = Z/W, alpha = 1 - exp(-A).
// This is baseline/fm_render.py:11-109 (and the reference kernel gaussianRayRasterizeCUDA,
// cuda_rasterizer/forward.cu:206-423) restricted to the tile's Gaussians.
#include <algorithm>

#include "fe_kernels.cuh"
#include "fe_tilerec.cuh"

namespace fe {

namespace {

template <int CH>
struct BlendSmem {
  TilePair buf[2][CH];      // record pairs: chunk c of a tile in buf[c & 1]
  GaussRec src[2 * CH];     // source records of the next chunk (TMA bulk copies), record r at src[r]
  uint64_t bar;             // completion of the source-record copies, one phase per chunk
  uint32_t tile;
  uint4 entry;              // the work-class list entry of the tile: x | y << 16, range, view
  uint32_t cls_base[kTileClasses + 1];  // first work index of each tile class (with `order`)
};

// Write a null record into slot `sl` (0 = .x, 1 = .y) of a pair: vsv = 1, psv = 0 (z = 0,
// masked), C = -inf (density 0).
__device__ __forceinline__ void null_slot(TilePair& p, int sl) {
#pragma unroll
  for (int i = 0; i < kRecFields; ++i) {
    float v = 0.f;
    if (i == 0) v = 1.f;
    if (i == 15) v = -INFINITY;
    if (sl == 0) p.f[i].x = v; else p.f[i].y = v;
  }
}

// Threads per CTA for a tile of TW x TH pixels with PX pixels per thread (PX consecutive pixels
// of one row, CW = TW/PX threads per row); GP record pairs per online-softmax group (one max
// update per group).
template <int TW, int TH, int PX, int CH, bool MANY>
struct BlendShape {
  static constexpr int NT = TW * TH / PX;
  // Resident CTAs per SM the register budget is sized for: 20 warps (640 threads) per SM leave the
  // 16x16 kernel 94 registers and no spills; at 24 warps it is held to 80 registers, spills a
  // little and runs about 1.3% slower. One-warp CTAs take 24 with groups of two pairs (80
  // registers), which the 8 KB of a 16-pair chunk allow and the 16 KB of a 32-pair one (13 CTAs)
  // do not. 8x8 tiles, 13 / 24 CTAs per SM: 16 views of 1000 Gaussians at 640x480 287 / 247 us per
  // forward, of 200 147 / 119, 1089 uneven views 1068 / 812.
  // MANY: 11 CTAs asked for (22 warps); 80 registers with 12 bytes spilled then let 12 run. Each is
  // a little slower, the SM faster, so it is for launches whose last tiles matter little (see
  // kManyTiles).
  static constexpr int MIN_CTAS = NT == 32 ? (CH <= 16 ? 24 : 13) : (MANY ? 704 : 640) / NT;
  static constexpr int CW = TW / PX;
  static constexpr int GP = PX >= 4 || NT == 32 ? 2 : 4;
  static_assert(TW % PX == 0, "PX must divide the tile width");
  static_assert(CH % GP == 0, "groups must tile a chunk");
  static_assert(NT >= GP, "enough threads to pad a chunk");
};

constexpr int kSplitPx = 2;  // pixels per thread of the split launches

// Initial running max: finite, far below any logit, so logit - max is never inf - inf.
constexpr float kNoLogit = -1e30f;

// Store a thread's PX consecutive pixels of one row (`room` pixels of the row remain from the
// first): one vector store when all PX lie inside the image and the address is aligned to it,
// else one store per pixel inside the image. The outputs may be pinned host memory mapped into
// the device's address space, where whole vectors keep the link's write rate.
template <int PX>
__device__ __forceinline__ void store_pixels(float* dst, const float (&x)[PX], int room) {
  const bool whole =
      room >= PX && (reinterpret_cast<uintptr_t>(dst) & (sizeof(float) * PX - 1)) == 0;
  if (PX == 4 && whole) {
    *reinterpret_cast<float4*>(dst) = make_float4(x[0], x[1], x[2 % PX], x[3 % PX]);
  } else if (PX == 2 && whole) {
    *reinterpret_cast<float2*>(dst) = make_float2(x[0], x[1 % PX]);
  } else {
#pragma unroll
    for (int k = 0; k < PX; ++k)
      if (k < room) dst[k] = x[k];
  }
}

// One group of GP record pairs for the thread's PX pixels: evaluate every logit, raise the running
// maxima once (rescaling W and Z), then accumulate. MASK applies the z > 0 mask to the logits.
template <int PX, int GP, bool MASK>
__device__ __forceinline__ void blend_group(const TilePair* grp, const f2_t (&DU)[PX], f2_t DV,
                                            f2_t DVSQ, f2_t B3, f2_t NB2, f2_t (&A2)[PX],
                                            f2_t (&W2)[PX], f2_t (&Z2)[PX], float (&m)[PX]) {
  f2_t ll[GP][PX], zz[GP][PX];
  float cmax[PX];
#pragma unroll
  for (int k = 0; k < PX; ++k) cmax[k] = -INFINITY;
#pragma unroll
  for (int q = 0; q < GP; ++q) {
    const ulonglong2* rp = reinterpret_cast<const ulonglong2*>(grp + q);
    const ulonglong2 r0 = rp[0], r1 = rp[1], r2 = rp[2], r3 = rp[3], r4 = rp[4];
    const ulonglong2 r5 = rp[5], r6 = rp[6], r7 = rp[7], r8 = rp[8];
    // V0..V5 = r0.x r0.y r1.x r1.y r2.x r2.y; P0..P2 = r3.x r3.y r4.x;
    // N0..N5 = r4.y r5.x r5.y r6.x r6.y r7.x; C = r7.y; cu = r8.x; cv = r8.y.
    // Row-constant parts first, shared by the thread's PX pixels.
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
      float sa, sb;
      f2_unpack(s2, sa, sb);
      A2[k] = add2(A2[k], f2_pack(ex2_approx(sa), ex2_approx(sb)));
      f2_t l = fma2(B3, s2, mul2(NB2, z));
      float l0, l1;
      f2_unpack(l, l0, l1);
      if (MASK) {
        float z0, z1;
        f2_unpack(z, z0, z1);
        l0 = z0 > 0.f ? l0 : -INFINITY;
        l1 = z1 > 0.f ? l1 : -INFINITY;
        l = f2_pack(l0, l1);
      }
      ll[q][k] = l;
      zz[q][k] = z;
      cmax[k] = max3f(cmax[k], l0, l1);
    }
  }
  // One branch for the thread's pixels (a branch each costs more than the rescaling by one of the
  // pixels whose maximum stays: 16 views 186.7 -> 184.0 us per pass, a 1280x720 view of 24000
  // Gaussians 323 -> 311).
  bool up = false;
#pragma unroll
  for (int k = 0; k < PX; ++k) up |= cmax[k] > m[k];
  if (up) {
#pragma unroll
    for (int k = 0; k < PX; ++k) {
      const float top = fmaxf(m[k], cmax[k]);
      const float sc = ex2_approx(m[k] - top);
      const f2_t S = f2_pack(sc, sc);
      W2[k] = mul2(W2[k], S);
      Z2[k] = mul2(Z2[k], S);
      m[k] = top;
    }
  }
#pragma unroll
  for (int k = 0; k < PX; ++k) {
    const f2_t M = f2_pack(m[k], m[k]);
#pragma unroll
    for (int q = 0; q < GP; ++q) {
      float d0, d1;
      f2_unpack(sub2(ll[q][k], M), d0, d1);
      const f2_t e = f2_pack(ex2_approx(d0), ex2_approx(d1));
      W2[k] = add2(W2[k], e);
      Z2[k] = fma2(e, zz[q][k], Z2[k]);
    }
  }
}

// nan_to_num with the limits of the reference's wrapper (fuzzy_ellipses/__init__.py:233-234): NaN
// and -inf become 0, +inf becomes `top`.
__device__ __forceinline__ float clean_value(float x, float top) {
  return x != x || x == -INFINITY ? 0.f : x == INFINITY ? top : x;
}

__device__ __forceinline__ float pixel_depth(float W, float Z) {
  return W > 0.f ? Z * rcp_approx(W) : 0.f;
}

// alpha = 1 - exp(-A): a Taylor polynomial below A = 1/64 (relative error under 1e-9), else from
// the hardware exp2 (absolute error under 3e-7).
__device__ __forceinline__ float pixel_alpha(float A) {
  return A < 0.015625f ? A * fmaf(A, fmaf(A, fmaf(A, -1.f / 24.f, 1.f / 6.f), -0.5f), 1.f)
                       : 1.f - ex2_approx(-A * kLog2e);
}

// Pieces of a tile of nk keys when a launch may cut tiles into up to `most`: consecutive keys, at
// least kMinPiece each; `per` receives a piece's keys (a multiple of 8, the last one fewer).
constexpr int kMinPiece = 64;
__device__ __forceinline__ int tile_pieces(int nk, int most, int& per) {
  const int p = max(1, min(most, nk / kMinPiece));
  per = p == 1 ? max(nk, 1) : ((nk + p - 1) / p + 7) & ~7;
  return (nk + per - 1) / per;
}

// CLEAN: the outputs go through clean_value. SPLIT: work index w is piece w / n_tiles of tile
// w % n_tiles (tile_end = n_tiles x the most pieces); a tile of several pieces leaves each one's
// sums (max logit, W, Z, A) per pixel in `part` for blend_merge_kernel.
template <int TW, int TH, int PX, int CH, bool CLEAN, bool SPLIT, bool MANY>
__global__ void __launch_bounds__(BlendShape<TW, TH, PX, CH, MANY>::NT,
                                  BlendShape<TW, TH, PX, CH, MANY>::MIN_CTAS) blend_fwd_kernel(
    ViewsArg va, uint32_t tile_begin, uint32_t tile_end, uint32_t* __restrict__ counter,
    const uint32_t* __restrict__ order, const uint64_t* __restrict__ keys,
    const GaussRec* __restrict__ recs, const uint2* __restrict__ ranges, float nb2, float beta3,
    float* __restrict__ depth, float* __restrict__ alpha, float* __restrict__ stats,
    int64_t stats_stride, uint32_t n_tiles, float4* __restrict__ part, Control* __restrict__ ctrl) {
  using Sh = BlendShape<TW, TH, PX, CH, MANY>;
  constexpr int GP = Sh::GP;
  __shared__ __align__(128) BlendSmem<CH> sm;

  const int tid = threadIdx.x;
  const int ly = tid / Sh::CW, cx = tid % Sh::CW;
  const float dv = ly - 0.5f * (TH - 1);
  const f2_t DV = f2_pack(dv, dv), DVSQ = f2_pack(dv * dv, dv * dv);
  const f2_t B3 = f2_pack(beta3, beta3), NB2 = f2_pack(nb2, nb2);
  // The thread's pixels are PX consecutive pixels of its row, so its outputs leave as one vector
  // store per plane.
  f2_t DU[PX];
#pragma unroll
  for (int k = 0; k < PX; ++k) {
    const float du = (cx * PX + k) - 0.5f * (TW - 1);
    DU[k] = f2_pack(du, du);
  }
  const f2_t ZERO2 = f2_pack(0.f, 0.f);

  constexpr int RC = 2 * CH;                     // records per chunk
  constexpr int RPT = (RC + Sh::NT - 1) / Sh::NT;  // records each thread stages and builds
  const float hw = 0.5f * (TW - 1), hh = 0.5f * (TH - 1);
  // Heaviest tiles first: with `order` (the tile-major binning's per-class tile lists over all
  // tiles [0, tile_end), uint4 entries: place in the view, first key, end key, view) work index w
  // of class c maps to entry w - cls_base[c] of its list, so the tiles taken last, which set the
  // kernel's tail, are the lightest, and a tile's range and view come with its id. The lists are
  // used only when they hold every tile exactly once (their counts sum to tile_end); else tiles go
  // in index order.
  chain_wait();
  if (tid == 0) {
    mbar_init(&sm.bar, 1);
    fence_mbar_init();
    if (order && tile_begin == 0) {
      uint32_t b = 0;
      for (int c = 0; c < kTileClasses; ++c) {
        sm.cls_base[c] = b;
        b += ctrl->tile_class[c];
      }
      sm.cls_base[kTileClasses] = b;
    }
  }
  __syncthreads();
  const bool listed = order && tile_begin == 0 && sm.cls_base[kTileClasses] == tile_end;
  uint32_t phase = 0;  // parity of the next completion of sm.bar

  // Work index of the CTA's first tile: its own index (the grid never exceeds the tiles), so the
  // launch does not start with every CTA contending for the counter; later tiles come from the
  // counter, offset by the grid.
  bool first = true;
  while (true) {
    if (tid < 32) {
      uint32_t w = tile_begin + blockIdx.x;
      if (!first) {
        if (tid == 0) w = atomicAdd(counter, 1u);
        w = tile_begin + gridDim.x + __shfl_sync(0xffffffffu, w, 0);
      }
      if (listed) {  // lane c looks at class c
        const uint32_t b = tid < kTileClasses ? sm.cls_base[tid] : 0u;
        const int c = 31 - __clz(__ballot_sync(0xffffffffu, tid < kTileClasses && b <= w));
        if (tid == c && w < tile_end)
          sm.entry = reinterpret_cast<const uint4*>(order)[list_entry(c, w - b, tile_end)];
      }
      if (tid == 0) sm.tile = w;
    }
    first = false;
    __syncthreads();
    const uint32_t item = sm.tile;
    if (item >= tile_end) break;
    const uint32_t piece = SPLIT ? item / n_tiles : 0u;
    const uint32_t tile = SPLIT ? item - piece * n_tiles : item;
    // With the work-class lists the entry carries the tile's place, range and view.
    int vi, tx, ty;
    uint2 rg;
    if (listed) {
      vi = (int)sm.entry.w;
      tx = (int)(sm.entry.x & 0xffffu);
      ty = (int)(sm.entry.x >> 16);
      rg = make_uint2(sm.entry.y, sm.entry.z);
    } else if (va.tile_ent) {
      const uint4 e = va.tile_ent[tile];
      vi = (int)e.w;
      tx = (int)(e.x & 0xffffu);
      ty = (int)(e.x >> 16);
      rg = make_uint2(e.y, e.z);
    } else {
      rg = ranges[tile];
      vi = view_of_tile(va, tile);
      const int gx = view_at(va, vi).gx;
      const int lt = (int)(tile - view_at(va, vi).tile_base);
      ty = lt / gx;
      tx = lt - ty * gx;
    }
    const GaussRec* vrec = recs + view_at(va, vi).rec_base;
    const float tcu = tx * TW + hw, tcv = ty * TH + hh;  // tile centre (pixels)

    bool whole = true;
    if (SPLIT) {
      int per;
      const uint32_t pieces = (uint32_t)tile_pieces((int)(rg.y - rg.x), (int)(tile_end / n_tiles),
                                                    per);
      if (piece > 0 && piece >= pieces) {
        __syncthreads();  // sm.tile is rewritten next iteration
        continue;
      }
      whole = pieces <= 1;
      rg.x += piece * (uint32_t)per;
      rg.y = min(rg.y, rg.x + (uint32_t)per);
    }
    // m starts finite (kNoLogit) so that logit - m is never (-inf) - (-inf); masked logits are
    // -inf and give weight 0.
    f2_t A2[PX], W2[PX], Z2[PX];
    float m[PX];
#pragma unroll
    for (int k = 0; k < PX; ++k) {
      A2[k] = ZERO2; W2[k] = ZERO2; Z2[k] = ZERO2;
      m[k] = kNoLogit;
    }
    if (rg.y > rg.x) {
      const int nk = (int)(rg.y - rg.x);
      const int nchunks = (nk + RC - 1) / RC;
      const uint64_t* tkeys = keys + rg.x;
      // Chunk c holds the tile's keys [c RC, c RC + RC); thread t stages and builds records
      // t, t + NT, ... of a chunk. The source records of chunk c + 1 arrive by TMA bulk copies
      // (96 B each, completing on sm.bar) while chunk c is evaluated; the Gaussian ids of chunk
      // c + 2 are read one chunk ahead of that. Copies into the staging buffer are issued only
      // after a barrier that every thread reaches after its wait for the previous chunk.
      uint32_t gid_next[RPT];
      auto stage = [&](int c, const uint32_t (&gid)[RPT]) {
        const int cnt = min(RC, nk - c * RC);
        fence_proxy_async_smem();  // this thread's reads of sm.src precede the copies into it
        if (tid == 0) mbar_arrive_expect_tx(&sm.bar, (uint32_t)(cnt * (int)sizeof(GaussRec)));
#pragma unroll
        for (int q = 0; q < RPT; ++q) {
          const int r = tid + q * Sh::NT;
          if (r < cnt) tma_bulk_g2s(&sm.src[r], vrec + gid[q], (uint32_t)sizeof(GaussRec), &sm.bar);
        }
      };
      auto wait_src = [&]() {
        const bool ok = mbar_wait_bounded(&sm.bar, phase);
        phase ^= 1u;
        return ok;
      };
      // A copy that did not land in time: flag it, give the outstanding copies one more bounded
      // wait and stop this CTA; the tile's outputs are left unwritten.
      auto give_up = [&]() {
        if (tid == 0) {
          atomicOr(&ctrl->error, FE_DEVERR_TIMEOUT);
          (void)mbar_wait_bounded(&sm.bar, phase ^ 1u);
        }
      };
      auto load_gids = [&](int c, uint32_t (&gid)[RPT]) {
#pragma unroll
        for (int q = 0; q < RPT; ++q) {
          const int r = tid + q * Sh::NT;
          gid[q] = (r < RC && c * RC + r < nk) ? (uint32_t)tkeys[c * RC + r] : 0u;
        }
      };
      // Build chunk c's record pairs from the staged source records (after the wait every
      // thread sees all of them; each builds its own) and null the slot past the tile's keys
      // that completes the last pair.
      auto build = [&](int c) {
        TilePair* pb = sm.buf[c & 1];
        const int cnt = min(RC, nk - c * RC);
        const int padded = (cnt + 1) & ~1;
#pragma unroll
        for (int q = 0; q < RPT; ++q) {
          const int r = tid + q * Sh::NT;
          if (r < cnt) {
            const GaussRec& g = sm.src[r];
            TileRec t;
            tile_record(g, tcu - g.uc, tcv - g.vc, hw, hh, t);
            const float* f = reinterpret_cast<const float*>(&t);
            float* dst = reinterpret_cast<float*>(&pb[r >> 1]) + (r & 1);
#pragma unroll
            for (int i = 0; i < kRecFields; ++i) dst[2 * i] = f[i];
          } else if (r < padded) {
            null_slot(pb[r >> 1], r & 1);
          }
        }
      };
      {
        // One staging buffer: chunk 1 is copied only once chunk 0 has been built from it.
        uint32_t g0[RPT];
        load_gids(0, g0);
        stage(0, g0);
        load_gids(1, g0);
        const bool ok = wait_src();
        build(0);
        if (__syncthreads_or(!ok)) {
          give_up();
          return;
        }
        if (nchunks > 1) stage(1, g0);
        load_gids(2, gid_next);
      }
      for (int c = 0; c < nchunks; ++c) {
        const int cnt = min(RC, nk - c * RC);
        const int pairs = (cnt + 1) >> 1;
        const TilePair* pb = sm.buf[c & 1];
        int j = 0;
        for (; j + GP <= pairs; j += GP) {
          // Uniform over the CTA: the z > 0 mask is only evaluated for groups holding a record
          // whose psv is not positive over the whole tile (null slots included).
          bool need_mask = false;
#pragma unroll
          for (int q = 0; q < GP; ++q) {
            const float2 fr = pb[j + q].f[18];
            need_mask |= !(fr.x != 0.f && fr.y != 0.f);
          }
          if (need_mask)
            blend_group<PX, GP, true>(&pb[j], DU, DV, DVSQ, B3, NB2, A2, W2, Z2, m);
          else
            blend_group<PX, GP, false>(&pb[j], DU, DV, DVSQ, B3, NB2, A2, W2, Z2, m);
        }
        // The pairs after the last whole group, in groups of two pairs, then one.
        for (; j < pairs;) {
          if (GP > 2 && j + 2 <= pairs) {
            const float2 f0 = pb[j].f[18], f1 = pb[j + 1].f[18];
            if (!(f0.x != 0.f && f0.y != 0.f && f1.x != 0.f && f1.y != 0.f))
              blend_group<PX, 2, true>(&pb[j], DU, DV, DVSQ, B3, NB2, A2, W2, Z2, m);
            else
              blend_group<PX, 2, false>(&pb[j], DU, DV, DVSQ, B3, NB2, A2, W2, Z2, m);
            j += 2;
          } else {
            const float2 f0 = pb[j].f[18];
            if (!(f0.x != 0.f && f0.y != 0.f))
              blend_group<PX, 1, true>(&pb[j], DU, DV, DVSQ, B3, NB2, A2, W2, Z2, m);
            else
              blend_group<PX, 1, false>(&pb[j], DU, DV, DVSQ, B3, NB2, A2, W2, Z2, m);
            j += 1;
          }
        }
        if (c + 1 < nchunks) {
          // Chunk c + 1: wait for its source records, build its pairs (buf[(c + 1) & 1] was last
          // read in chunk c - 1), publish them, then stage chunk c + 2.
          const bool ok = wait_src();
          build(c + 1);
          if (__syncthreads_or(!ok)) {
            give_up();
            return;
          }
          if (c + 2 < nchunks) {
            stage(c + 2, gid_next);
            load_gids(c + 3, gid_next);
          }
        }
      }
    }

    const ViewDev& V = view_at(va, vi);
    const int v = ty * TH + ly;
    const int u0 = tx * TW + cx * PX;
    if (SPLIT && !whole) {
      float4* dst = part + (int64_t)item * (TW * TH) + ly * TW + cx * PX;
#pragma unroll
      for (int k = 0; k < PX; ++k) {
        float a0, a1, w0, w1, z0, z1;
        f2_unpack(A2[k], a0, a1);
        f2_unpack(W2[k], w0, w1);
        f2_unpack(Z2[k], z0, z1);
        dst[k] = make_float4(m[k], w0 + w1, z0 + z1, a0 + a1);
      }
    } else if (v < V.H) {
      float dep[PX], alp[PX], wsum[PX], asum[PX];
#pragma unroll
      for (int k = 0; k < PX; ++k) {
        float a0, a1, w0, w1, z0, z1;
        f2_unpack(A2[k], a0, a1);
        f2_unpack(W2[k], w0, w1);
        f2_unpack(Z2[k], z0, z1);
        const float A = a0 + a1, W = w0 + w1, Z = z0 + z1;
        dep[k] = pixel_depth(W, Z);
        alp[k] = pixel_alpha(A);
        wsum[k] = W;
        asum[k] = A;
        if (CLEAN) {
          dep[k] = clean_value(dep[k], 10.f);
          alp[k] = clean_value(alp[k], 1.f);
        }
      }
      const int64_t pix = V.pix_base + (int64_t)v * V.W + u0;
      store_pixels<PX>(depth + pix, dep, V.W - u0);
      store_pixels<PX>(alpha + pix, alp, V.W - u0);
      if (stats) {
        store_pixels<PX>(stats + pix, m, V.W - u0);
        store_pixels<PX>(stats + stats_stride + pix, wsum, V.W - u0);
        store_pixels<PX>(stats + 2 * stats_stride + pix, asum, V.W - u0);
      }
    }
    __syncthreads();  // sm.tile is rewritten next iteration
  }
}

// The pixels of the tiles that were blended in pieces: a thread per pixel merges the pieces' sums
// in piece order. One block per tile; the tiles of a single piece are already written.
template <int TW, int TH>
__global__ void __launch_bounds__(TW * TH) blend_merge_kernel(
    ViewsArg va, uint32_t n_tiles, int most, const uint2* __restrict__ ranges,
    const float4* __restrict__ part, float* __restrict__ depth, float* __restrict__ alpha,
    float* __restrict__ stats, int64_t stats_stride) {
  chain_wait();
  const uint32_t tile = blockIdx.x;
  const uint2 rg = ranges[tile];
  int per;
  const int pieces = tile_pieces((int)(rg.y - rg.x), most, per);
  if (pieces <= 1) return;
  const ViewDev& V = view_at(va, view_of_tile(va, tile));
  const int lt = (int)(tile - V.tile_base);
  const int u = (lt % V.gx) * TW + (int)threadIdx.x % TW;
  const int v = (lt / V.gx) * TH + (int)threadIdx.x / TW;
  if (u >= V.W || v >= V.H) return;
  float m = kNoLogit, W = 0.f, Z = 0.f, A = 0.f;
#pragma unroll 4
  for (int p = 0; p < pieces; ++p) {
    const float4 x = part[((int64_t)p * n_tiles + tile) * (TW * TH) + threadIdx.x];
    const float top = fmaxf(m, x.x), a = ex2_approx(m - top), b = ex2_approx(x.x - top);
    W = fmaf(W, a, x.y * b);
    Z = fmaf(Z, a, x.z * b);
    A += x.w;
    m = top;
  }
  const int64_t pix = V.pix_base + (int64_t)v * V.W + u;
  depth[pix] = pixel_depth(W, Z);
  alpha[pix] = pixel_alpha(A);
  if (stats) {
    stats[pix] = m;
    stats[stats_stride + pix] = W;
    stats[2 * stats_stride + pix] = A;
  }
}

template <int TW, int TH, int PX, int CH, bool CLEAN = false, bool MANY = false>
void launch_tiles(const ViewsArg& va, int64_t tile_begin, int64_t tile_end, uint32_t* counter,
                  const uint32_t* order, const uint64_t* keys, const GaussRec* recs,
                  const uint2* ranges, float nb2, float beta3, float* depth, float* alpha,
                  float* stats, int64_t stats_stride, Control* ctrl, cudaStream_t st) {
  constexpr int NT = BlendShape<TW, TH, PX, CH, MANY>::NT;
  constexpr auto kern = blend_fwd_kernel<TW, TH, PX, CH, CLEAN, false, MANY>;
  const int64_t grid = std::min<int64_t>(tile_end - tile_begin, resident_ctas<kern>(NT));
  // (a host call's bands, with counters of their own, follow an event or one another)
  launch_chained(va.chain && counter == &ctrl->next_tile, kern, (unsigned)grid, NT, st, va,
                 (uint32_t)tile_begin, (uint32_t)tile_end, counter, order, keys, recs, ranges, nb2,
                 beta3, depth, alpha, stats, stats_stride, 0u, nullptr, ctrl);
}

template <int TW, int TH>
void launch_split(const ViewsArg& va, int64_t n_tiles, int pieces, const uint64_t* keys,
                  const GaussRec* recs, const uint2* ranges, float nb2, float beta3, float* depth,
                  float* alpha, float* stats, int64_t stats_stride, float4* part, Control* ctrl,
                  cudaStream_t st) {
  constexpr int PX = kSplitPx, CH = TW * TH / PX == 32 ? 16 : 32;
  constexpr int NT = BlendShape<TW, TH, PX, CH, false>::NT;
  constexpr auto kern = blend_fwd_kernel<TW, TH, PX, CH, false, true, false>;
  const int64_t items = n_tiles * pieces;
  const int64_t grid = std::min<int64_t>(items, resident_ctas<kern>(NT));
  launch_chained(va.chain, kern, (unsigned)grid, NT, st, va, 0u, (uint32_t)items,
                 &ctrl->next_tile, nullptr, keys, recs, ranges, nb2, beta3, depth, alpha, stats,
                 stats_stride, (uint32_t)n_tiles, part, ctrl);
  launch_chained(va.chain, blend_merge_kernel<TW, TH>, (unsigned)n_tiles, TW * TH, st, va,
                 (uint32_t)n_tiles, pieces, ranges, part, depth, alpha, stats, stats_stride);
}

// Tiles from which 24 warps per SM finish sooner than 20 faster ones: 7 per CTA. Forward, 20 / 24
// warps: 1089 uneven views (122 K tiles) 649 / 633 us, 60 scenes (28 K) 214.3 / 212.5, 16 views of
// 640x480 (19200) 179.2 / 178.7, of 200 Gaussians 77.5 / 76.0, 32 of 20 Gaussians 84.1 / 80.0; one
// of 1280x720 (3600) 260 / 275. Launches that store straight into host memory wait for the link and
// lose 0.5%: they ask for the chunk size they would get.
constexpr int64_t kManyTiles = 8 * 152 * 11;

template <int TW, int TH, int PX>
void launch_chunk(int chunk, const ViewsArg& va, int64_t tile_begin, int64_t tile_end,
                  uint32_t* counter, const uint32_t* order, const uint64_t* keys,
                  const GaussRec* recs, const uint2* ranges, float nb2, float beta3, float* depth,
                  float* alpha, float* stats, int64_t stats_stride, Control* ctrl,
                  cudaStream_t st) {
  if (chunk == 8)
    launch_tiles<TW, TH, PX, 8>(va, tile_begin, tile_end, counter, order, keys, recs, ranges, nb2,
                                beta3, depth, alpha, stats, stats_stride, ctrl, st);
  else if (chunk == 16 || (chunk != 32 && TW * TH / PX == 32))
    launch_tiles<TW, TH, PX, 16>(va, tile_begin, tile_end, counter, order, keys, recs, ranges,
                                 nb2, beta3, depth, alpha, stats, stats_stride, ctrl, st);
  else if (PX == 4 && chunk == 0 && tile_end - tile_begin >= kManyTiles)
    launch_tiles<TW, TH, PX, 32, false, PX == 4>(va, tile_begin, tile_end, counter, order, keys,
                                                 recs, ranges, nb2, beta3, depth, alpha, stats,
                                                 stats_stride, ctrl, st);
  else
    launch_tiles<TW, TH, PX, 32>(va, tile_begin, tile_end, counter, order, keys, recs, ranges,
                                 nb2, beta3, depth, alpha, stats, stats_stride, ctrl, st);
}

}  // namespace

namespace {

void blend_dispatch(const ViewsArg& va, int tile_w, int tile_h, int px, int chunk,
                    int64_t tile_begin, int64_t tile_end, uint32_t* counter, const uint32_t* order,
                    const uint64_t* keys, const GaussRec* recs, const uint2* ranges, float beta2,
                    float beta3, float* depth, float* alpha, float* stats, int64_t stats_stride,
                    Control* ctrl, cudaStream_t st) {
  if (tile_end <= tile_begin) return;
  const float nb2 = -beta2 * kLog2e;
#define FE_BLEND(TW_, TH_, PX_)                                                                 \
  launch_chunk<TW_, TH_, PX_>(chunk, va, tile_begin, tile_end, counter, order, keys, recs, ranges, \
                              nb2, beta3, depth, alpha, stats, stats_stride, ctrl, st)
  if (tile_w == 8 && tile_h == 8) {
    if (px == 1) FE_BLEND(8, 8, 1); else FE_BLEND(8, 8, 2);
  } else if (tile_w == 32 && tile_h == 8) {
    if (px == 1) FE_BLEND(32, 8, 1); else if (px == 2) FE_BLEND(32, 8, 2); else FE_BLEND(32, 8, 4);
  } else {
    if (px == 1) FE_BLEND(16, 16, 1); else if (px == 2) FE_BLEND(16, 16, 2); else FE_BLEND(16, 16, 4);
  }
#undef FE_BLEND
}

}  // namespace

// Pixels per thread: px in {1, 2, 4} (8x8 tiles: 1, 2); 0 selects the default for the tile.
// Chunk: record pairs per shared-memory stage, 8, 16 or 32; 0 selects 32 (one-warp CTAs: 16).
void launch_blend_fwd_band(const ViewsArg& va, int tile_w, int tile_h, int px, int chunk,
                           int64_t tile_begin, int64_t tile_end, uint32_t* counter,
                           const uint64_t* keys, const GaussRec* recs, const uint2* ranges,
                           float beta2, float beta3, float* depth, float* alpha, float* stats,
                           int64_t stats_stride, Control* ctrl, cudaStream_t st) {
  blend_dispatch(va, tile_w, tile_h, px, chunk, tile_begin, tile_end, counter, nullptr, keys, recs,
                 ranges, beta2, beta3, depth, alpha, stats, stats_stride, ctrl, st);
}

int blend_pieces(int tile_w, int tile_h, int px, int chunk, int64_t n_tiles, int64_t max_n) {
  if ((px != 0 && px != kSplitPx) || (px == 0 && !(tile_w == 8 && tile_h == 8)) ||
      (chunk != 0 && chunk != 32) || n_tiles <= 0)
    return 1;
  // A launch of few tiles leaves SMs idle and lasts as long as its heaviest tile (the keys of a
  // tile are blended one after the other). Tiles are cut until the pieces could fill the GPU (CTAs
  // as BlendShape sizes them) twice over, more often the more keys per tile the view can hold; a
  // piece has at least 128 keys in the densest tile there can be (64 in fact: tile_pieces). Per
  // call, whole / cut: 2600 Gaussians at 64x64 158 / 57 us, 4378 at 73x419 202 / 96, 1422 at
  // 293x157 96 / 64, 931 at 347x170 67 / 52, 20000 at 300x400 260 / 168, 8273 at 621x573 172 / 153;
  // with more pieces where they hold fewer keys, 1100 at 640x480 53 / 58, 1000 at 637x479 75 / 80.
  const int64_t cta = 152 * std::min(16, 640 / (tile_w * tile_h / kSplitPx));
  const int64_t most = cta * (max_n < 2 * n_tiles || max_n <= 1024 ? 2 : max_n <= 4096 ? 4 : 8);
  int pieces = 1;
  while (pieces < 32 && 2 * pieces * n_tiles <= most && 2 * pieces * 128 <= max_n) pieces *= 2;
  return pieces;
}

void launch_blend_fwd(const ViewsArg& va, int tile_w, int tile_h, int px, int chunk,
                      int64_t n_tiles, const uint32_t* order, int pieces, float4* part,
                      const uint64_t* keys,
                      const GaussRec* recs, const uint2* ranges, float beta2, float beta3,
                      float* depth, float* alpha, float* stats, int64_t stats_stride,
                      Control* ctrl, cudaStream_t st) {
  if (pieces > 1 && part) {
    const float nb2 = -beta2 * kLog2e;
    auto go = [&](auto launch) {
      launch(va, n_tiles, pieces, keys, recs, ranges, nb2, beta3, depth, alpha, stats, stats_stride,
             part, ctrl, st);
    };
    if (tile_w == 8 && tile_h == 8) go(launch_split<8, 8>);
    else if (tile_w == 32 && tile_h == 8) go(launch_split<32, 8>);
    else go(launch_split<16, 16>);
    return;
  }
  blend_dispatch(va, tile_w, tile_h, px, chunk, 0, n_tiles, &ctrl->next_tile, order, keys, recs,
                 ranges, beta2, beta3, depth, alpha, stats, stats_stride, ctrl, st);
}

void launch_blend_fwd_clean(const ViewsArg& va, int64_t n_tiles, const uint64_t* keys,
                            const GaussRec* recs, const uint2* ranges, float beta2, float beta3,
                            float* depth, float* alpha, Control* ctrl, cudaStream_t st) {
  if (n_tiles <= 0) return;
  launch_tiles<8, 8, 2, 16, true>(va, 0, n_tiles, &ctrl->next_tile, nullptr, keys, recs, ranges,
                                  -beta2 * kLog2e, beta3, depth, alpha, nullptr, 0, ctrl, st);
}

}  // namespace fe

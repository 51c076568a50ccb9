// ordered.cuh -- imaging with every point's sum in submission order (the plain
// and the compat kernel), sm_100a.
//
// A block of 256 threads images 32 depths x 8/SPLIT cdps.  Per chunk of 256
// traces, each thread decides one trace for the whole tile (aperture, table
// coverage, the dip bound of tile.cuh) and the kept ones are listed in shared
// memory in submission order.  The points then run over the list.
//
// SPLIT > 1: SPLIT warps share a column of 32 points.  Each evaluates its share
// of a round of kept traces into shared memory, and one warp adds the round's
// values in order: evaluation, which is all the work, is parallel over the
// traces, and each point's sum is still that of one thread running over them.
#pragma once

#include <type_traits>

#include "common.cuh"

namespace qpsdm {

constexpr int kOrdChunk = 256, kOrdShare = 8;  // traces per chunk; per warp and round

template <int SPLIT>
struct OrderedSmem {
  int4 rec[kOrdChunk];
  float4 geo[kOrdChunk];  // source and receiver, relative to the line
  float2 wgt[kOrdChunk];  // surface weights of the receiver (plain kernel)
  unsigned mask[8];       // kept traces of the chunk, one bit each
  int wpos[9];            // kept traces before word w
  // a round's values of each column and which points have one (double-buffered)
  float val[SPLIT > 1 ? 2 : 1][SPLIT > 1 ? 8 * kOrdShare : 1][32];
  unsigned has[SPLIT > 1 ? 2 : 1][SPLIT > 1 ? 8 * kOrdShare : 1];
};

// keep(i, rec, geo, wgt): whether trace i is kept for the tile, and its record;
// eval(k, value): whether the thread's point takes list entry k; add(value) in
// submission order.  Called by all 256 threads of the block; `act`: the
// thread's point takes part.
template <int SPLIT, typename Keep, typename Eval, typename Add>
__device__ __forceinline__ void ordered_walk(OrderedSmem<SPLIT> &sm, int ntr, bool act,
                                             const Keep &keep, const Eval &eval, const Add &add) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int c0 = 0; c0 < ntr; c0 += kOrdChunk) {
    __syncthreads();  // the list is rewritten
    int4 r;
    float4 g;
    float2 h;
    const bool k = c0 + tid < ntr && keep(c0 + tid, r, g, h);
    const unsigned bits = __ballot_sync(0xffffffffu, k);
    if (lane == 0) sm.mask[warp] = bits;
    __syncthreads();
    int before = 0, nkept = 0;
#pragma unroll
    for (int w = 0; w < 8; ++w) {
      const int c = __popc(sm.mask[w]);
      if (w < warp) before += c;
      nkept += c;
    }
    if (k) {
      const int at = before + __popc(bits & ((1u << lane) - 1u));
      sm.rec[at] = r;
      sm.geo[at] = g;
      sm.wgt[at] = h;
    }
    __syncthreads();
    if (SPLIT == 1) {
      if (act)
        for (int i = 0; i < nkept; ++i) {
          float v;
          if (eval(i, v)) add(v);
        }
      continue;
    }
    constexpr int R = SPLIT * kOrdShare;  // traces per round
    const int share = warp % SPLIT, row0 = (warp / SPLIT) * R;
    int buf = 0;
    for (int k0 = 0; k0 < nkept; k0 += R, buf ^= 1) {
#pragma unroll 1
      for (int j = 0; j < kOrdShare; ++j) {
        const int i = share * kOrdShare + j;
        if (k0 + i >= nkept) break;
        float v = 0.0f;
        const bool p = act && eval(k0 + i, v);
        const unsigned m = __ballot_sync(0xffffffffu, p);
        if (p) sm.val[buf][row0 + i][lane] = v;
        if (lane == 0) sm.has[buf][row0 + i] = m;
      }
      __syncthreads();
      if (share == 0) {  // the other warps go on with the next round
        const int n = min(R, nkept - k0);
        for (int i = 0; i < n; ++i)
          if ((sm.has[buf][row0 + i] >> lane) & 1u) add(sm.val[buf][row0 + i][lane]);
      }
    }
  }
}

// Calls f with the number of warps per column: the fewest that give the GPU four
// times the warps it holds (sm_warps per SM: the kernel's occupancy), so that
// uneven blocks balance.  More share the tile's per-trace decisions between
// fewer points.  Measured, warps per column 1 / 2 / 4 / 8 -- compat (32 warps
// an SM): 1024 x 600 points 2.18 / 2.32 / 2.61 / 3.91 ms, 512 x 400 5.13 / 3.91 /
// 3.35 / 4.41, 300 x 250 2.55 / 1.68 / 1.05 / 1.00, 128 x 100 0.62 / 0.43 / 0.23 /
// 0.13; plain (16 warps an SM): 2.69 / 3.24 / 3.74 / 4.95, 5.78 / 5.60 / 6.08 / 7.19,
// 3.38 / 2.28 / 1.64 / 1.79, 0.76 / 0.56 / 0.31 / 0.18 ms.
template <typename F>
void ordered_by_split(int nzi, int nxb, int sm_warps, const F &f) {
  int dev = 0, nsm = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  const int64_t warps = (int64_t)((nzi + 31) / 32) * nxb, want = 4ll * nsm * sm_warps;
  if (warps >= want)
    f(std::integral_constant<int, 1>());
  else if (2 * warps >= want)
    f(std::integral_constant<int, 2>());
  else if (4 * warps >= want)
    f(std::integral_constant<int, 4>());
  else
    f(std::integral_constant<int, 8>());
}

// The pass/fail side of a dip limit without the division: with uz > 0, the
// sign of fma(-c, uz, ux) is that of ux / uz - c exactly, so a non-positive one
// means ux / uz <= c, and then the rounded quotient is <= c too.
__device__ __forceinline__ float dip_side(float ux, float uz, float c) {
  return __fmaf_rn(-c, uz, ux);
}

struct DipLimits {
  float x1, x2, y1, y2;      // limits
  float x1c, x2c, y1c, y2c;  // limits widened by the taper zone
  bool wide;  // each limit lies strictly inside its widened one
};

// Dip test and taper of a pair, w = the product of the taper factors: the
// bits of
//   tanx = ux / uz, tany = uy / uz
//   tanx > x1c && tanx < x2c && tany > y1c && tany < y2c  (else false)
//   w = 1; if (tanx < x1) w *= (tanx - x1c) / (x1 - x1c); if (tanx > x2) ...
// with the divisions only where their value is used: inside a taper zone.  A
// quotient at or inside the limit itself passes the widened one.
__device__ __forceinline__ bool dip_taper(float ux, float uy, float uz, const DipLimits &d,
                                          float &w) {
  // a NaN tangent (0/0 at z = 0) fails like any other: !(a > b)
  if (!(dip_side(ux, uz, d.x1c) > 0.0f && dip_side(ux, uz, d.x2c) < 0.0f &&
        dip_side(uy, uz, d.y1c) > 0.0f && dip_side(uy, uz, d.y2c) < 0.0f))
    return false;
  w = 1.0f;
  if (!d.wide || dip_side(ux, uz, d.x1) < 0.0f || dip_side(ux, uz, d.x2) > 0.0f) {
    const float tanx = __fdiv_rn(ux, uz);
    if (!(tanx > d.x1c && tanx < d.x2c)) return false;
    if (tanx < d.x1)
      w = __fmul_rn(w, __fdiv_rn(__fsub_rn(tanx, d.x1c), __fsub_rn(d.x1, d.x1c)));
    if (tanx > d.x2)
      w = __fmul_rn(w, __fdiv_rn(__fsub_rn(d.x2c, tanx), __fsub_rn(d.x2c, d.x2)));
  }
  if (!d.wide || dip_side(uy, uz, d.y1) < 0.0f || dip_side(uy, uz, d.y2) > 0.0f) {
    const float tany = __fdiv_rn(uy, uz);
    if (!(tany > d.y1c && tany < d.y2c)) return false;
    if (tany < d.y1)
      w = __fmul_rn(w, __fdiv_rn(__fsub_rn(tany, d.y1c), __fsub_rn(d.y1, d.y1c)));
    if (tany > d.y2)
      w = __fmul_rn(w, __fdiv_rn(__fsub_rn(d.y2c, tany), __fsub_rn(d.y2c, d.y2)));
  }
  return true;
}

}  // namespace qpsdm

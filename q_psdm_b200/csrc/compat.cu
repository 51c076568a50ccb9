// compat.cu -- the reference-compatible imaging path on sm_100a.
//
//   k_gate      psdm_kernel's per-trace geometry gate (src/q-psdm.cu:2107-2171)
//   k_spectra   psdm_kernel's preprocessing: t^2 gain, tapers, two r2c
//               windows, -i*w (src/q-psdm.cu:2174-2219, psdmpkg.cc:208-231)
//   k_image_compat  image_depth_gpu with the reference's ts = tg = 1 stub
//               (src/q-psdm.cu:2246-2379), batched over traces
//
// Rounding: every operation that feeds an index, a mask or the image uses an
// explicit IEEE intrinsic (__fadd_rn, __fdiv_rn, __fsqrt_rn, __dadd_rn, ...)
// so that nothing is contracted into an FMA or approximated; a plain C
// restatement built with -ffp-contract=off computes the same bits.
#include "common.cuh"
#include "fft.cuh"
#include "internal.h"
#include "ordered.cuh"
#include "tile.cuh"

namespace qpsdm {

// ---------------------------------------------------------------------------
// Gate: one thread per trace.
// ---------------------------------------------------------------------------
__device__ __forceinline__ bool gate_trace(const uint8_t *__restrict__ rec, int rec_bytes,
                                           int itr, int be, const GateArgs &g,
                                           int *__restrict__ ints, float *__restrict__ geom,
                                           unsigned *err) {
  const uint8_t *r = rec + (size_t)itr * rec_bytes;
  int *o = ints + (size_t)itr * kGateInts;
  float *f = geom + (size_t)itr * kGateF;
#pragma unroll
  for (int i = 0; i < kGateInts; ++i) o[i] = 0;
#pragma unroll
  for (int i = 0; i < kGateF; ++i) f[i] = 0.0f;

  const double sx = __dmul_rn((double)su_i32(r, kOffSx, be), g.scaled);
  const double sy = __dmul_rn((double)su_i32(r, kOffSy, be), g.scaled);
  const double gx = __dmul_rn((double)su_i32(r, kOffGx, be), g.scaled);
  const double gy = __dmul_rn((double)su_i32(r, kOffGy, be), g.scaled);
  if (sx < g.fxv1 || sx > g.exv1 || gx < g.fxv1 || gx > g.exv1 ||
      sy < g.fyv1 || sy > g.eyv1 || gy < g.fyv1 || gy > g.eyv1) {
    o[0] = kRejBbox;
    return false;
  }
  const double ddx = __dsub_rn(gx, sx), ddy = __dsub_rn(gy, sy);
  const double offset = (double)__fsqrt_rn(
      __double2float_rn(__dadd_rn(__dmul_rn(ddx, ddx), __dmul_rn(ddy, ddy))));
  const int cdpx = __double2int_rz(__dadd_rn(
      __ddiv_rn(__dsub_rn(__dmul_rn(__dadd_rn(sx, gx), 0.5), g.fxi), (double)g.dxi), 0.5));
  const int cdpy = __double2int_rz(__dadd_rn(
      __ddiv_rn(__dsub_rn(__dmul_rn(__dadd_rn(sy, gy), 0.5), g.cyi), (double)g.dyi), 0.5));
  int iaz = 0;
  if (offset > 1.0) {
    float cosx = fabsf(__double2float_rn(__ddiv_rn(ddx, offset)));
    if (__dmul_rn(ddx, ddy) < 0.0) cosx = -cosx;
    const float c1 = __double2float_rn(__dsub_rn(1.0, (double)cosx));
    int i = __float2int_rz(__fdiv_rn(c1, g.eps));
    if (i < 0 || i >= g.naztab) {  // cannot happen for |cos| <= 1; never read out of bounds
      atomicOr(err, kErrIaz);
      i = i < 0 ? 0 : g.naztab - 1;
    }
    iaz = g.iaztab[i];
  }
  o[1] = cdpx;
  o[2] = cdpy;
  o[3] = iaz;
  int nx1 = g.az[0][iaz], nx2 = g.az[1][iaz];
  int ny1 = g.az[2][iaz], ny2 = g.az[3][iaz];
  if (g.cap) {  // the trace's own aperture caps the offset group's
    const int cx = g.cap[2 * (size_t)itr], cy = g.cap[2 * (size_t)itr + 1];
    nx1 = min(nx1, cx);
    nx2 = min(nx2, cx);
    ny1 = min(ny1, cy);
    ny2 = min(ny2, cy);
  }
  if (cdpy > ny1 || cdpy < -ny2) {
    o[0] = kRejY;
    return false;
  }
  // Columns cdpx-nx1 .. cdpx+nx2-1 clipped to the block; every column starts
  // at depth 0 and columns exist only when nzi > 10 (src/q-psdm.cu:2155-2171).
  int first = cdpx - nx1, last = cdpx + nx2 - 1;
  if (first < g.ixstart) first = g.ixstart;
  if (last > g.ixend - 1) last = g.ixend - 1;
  const int ntibeg = (g.nzi > 10 && last >= first) ? last - first + 1 : 0;
  if (ntibeg == 0) {
    o[0] = kRejCols;
    return false;
  }
  o[0] = kAccepted;
  o[4] = first;
  o[5] = last;
  o[6] = ntibeg;
  o[7] = 0;
  f[0] = __double2float_rn(__dsub_rn(sx, g.fxi));
  f[1] = __double2float_rn(__dsub_rn(sy, g.cyi));
  f[2] = __double2float_rn(__dsub_rn(gx, g.fxi));
  f[3] = __double2float_rn(__dsub_rn(gy, g.cyi));
  return true;
}

__global__ void k_gate(const uint8_t *__restrict__ rec, int rec_bytes, int ntr,
                       int be, GateArgs g, int *__restrict__ ints,
                       float *__restrict__ geom, unsigned *err,
                       unsigned long long *__restrict__ nacc) {
  const int itr = blockIdx.x * blockDim.x + threadIdx.x;
  // accepted traces of the block, one atomic per warp (graph replays count too)
  const bool accepted = itr < ntr && gate_trace(rec, rec_bytes, itr, be, g, ints, geom, err);
  const unsigned ballot = __ballot_sync(0xffffffffu, accepted);
  if (nacc && (threadIdx.x & 31) == 0 && ballot)
    atomicAdd(nacc, (unsigned long long)__popc(ballot));
}

int launch_gate(const uint8_t *d_rec, int rec_bytes, int ntr, int be,
                const GateArgs &g, int *d_ints, float *d_geom, unsigned *d_err,
                unsigned long long *d_nacc, cudaStream_t s) {
  if (ntr <= 0) return QPSDM_OK;
  k_gate<<<(ntr + 127) / 128, 128, 0, s>>>(d_rec, rec_bytes, ntr, be, g, d_ints,
                                           d_geom, d_err, d_nacc);
  return cudaGetLastError() == cudaSuccess ? QPSDM_OK : QPSDM_ECUDA;
}

// ---------------------------------------------------------------------------
// Spectra: one CTA per accepted trace, its two windows transformed together
// (fft.cuh).
// ---------------------------------------------------------------------------

// Gained sample j of the trace, then the full-trace end taper applied in the
// reference's order (src/psdmpkg.cc:221-228: head factor at iteration j, tail
// factor at iteration n-1-j; the earlier iteration multiplies first).
__device__ __forceinline__ float tapered_sample(float v, int j, int n,
                                                const float *tap) {
  const int head = j, tail = n - 1 - j;
  const bool h = head < 200, t = tail < 200;
  if (h && t) {
    if (head <= tail) {
      v = __fmul_rn(v, tap[head]);
      v = __fmul_rn(v, tap[tail]);
    } else {
      v = __fmul_rn(v, tap[tail]);
      v = __fmul_rn(v, tap[head]);
    }
  } else if (h) {
    v = __fmul_rn(v, tap[head]);
  } else if (t) {
    v = __fmul_rn(v, tap[tail]);
  }
  return v;
}

__device__ __forceinline__ float gained(float v, int it, float dt) {
  const float t = __fmul_rn((float)it, dt);
  if ((double)t < 0.1) return __double2float_rn(__dmul_rn((double)v, 0.1 * 0.1));
  return __fmul_rn(v, __fmul_rn(t, t));
}

// Sample i of window [itb, itb + nsb) of the trace, tapered again to the window.
__device__ __forceinline__ float window_sample(const uint8_t *r, int be, const SpectraArgs &a,
                                               int itb, int i) {
  const int j = itb + i;
  float v = 0.0f;
  if (j >= 0 && j < a.ntl)
    v = tapered_sample(gained(su_sample(r, j, be), j, a.dt), j, a.ntl, a.taper200);
  return tapered_sample(v, i, a.nsb, a.taper200);
}

template <int MODE>
__global__ void __launch_bounds__(kFftMaxThreads, 2)
    k_spectra(const uint8_t *__restrict__ rec, int rec_bytes, int be,
              const int *__restrict__ ints, const __grid_constant__ SpectraArgs a,
              const __grid_constant__ FftPlan p, float *__restrict__ re,
              float *__restrict__ im) {
  const int itr = blockIdx.x;
  if (ints[(size_t)itr * kGateInts] != kAccepted) return;
  extern __shared__ float4 pbuf[];
  const uint8_t *r = rec + (size_t)itr * rec_bytes;
  for (int j = threadIdx.x; j < p.m; j += blockDim.x)
    pbuf[pfa_slot<MODE>(j)] = make_float4(
        window_sample(r, be, a, a.itb1, 2 * j), window_sample(r, be, a, a.itb2, 2 * j),
        window_sample(r, be, a, a.itb1, 2 * j + 1), window_sample(r, be, a, a.itb2, 2 * j + 1));
  __syncthreads();
  const float4 *Z = fft_passes<MODE>(pbuf, p);
  float *ro = re + (size_t)itr * 2 * a.nww, *io = im + (size_t)itr * 2 * a.nww;
  for (int iw = threadIdx.x; iw < a.nww; iw += blockDim.x) {
    // bin k <= m from Z[k] and Z[m-k]
    const int k = iw + a.nf1;
    C2 X, unused;
    pfa_rfft_bins(pfa_ld(Z, pfa_slot<MODE>(k == p.m ? 0 : k)),
                  pfa_ld(Z, pfa_slot<MODE>(k == 0 ? 0 : p.m - k)), __ldg(p.tw_n + k), X, unused);
    const float2 xr = f2_unpack(X.re), xi = f2_unpack(X.im);
    const float w = a.omega[iw];
    ro[iw] = __fmul_rn(xi.x, w);
    io[iw] = -__fmul_rn(xr.x, w);
    ro[a.nww + iw] = __fmul_rn(xi.y, w);
    io[a.nww + iw] = -__fmul_rn(xr.y, w);
  }
}

int launch_spectra(const uint8_t *d_rec, int rec_bytes, int ntr, int be,
                   const int *d_ints, const SpectraArgs &a, float *d_re,
                   float *d_im, cudaStream_t s) {
  if (ntr <= 0) return QPSDM_OK;
  FftPlan p;
  std::string err;
  int rc = fft_plan(a.nsb, &p, &err);
  if (rc) return rc;
  return fft_by_mode(p, [&](auto mode) {
    auto kern = k_spectra<decltype(mode)::value>;
    const size_t sm = fft_smem_bytes(p);
    if ((rc = fft_set_smem_attr((const void *)kern, sm))) return rc;
    kern<<<ntr, p.threads, sm, s>>>(d_rec, rec_bytes, be, d_ints, a, p, d_re, d_im);
    return cudaGetLastError() == cudaSuccess ? (int)QPSDM_OK : (int)QPSDM_ECUDA;
  });
}

// ---------------------------------------------------------------------------
// Stub imaging: traces in submission order at every point (ordered.cuh).
//
// Bound by issued instructions (IEEE square roots, divisions, one double
// reciprocal per imaged pair).  9,216 traces into a 512 x 400 line (1.1e9
// point-traces): 10.0 ms with 11 divisions and a double one for every pair;
// 3.35 ms with the tile's dip bound, the tangents' divisions only inside the
// taper zones, one reciprocal for the six divisions by the receiver distance
// and the source terms kept from trace to trace.  1,024 traces into a
// 128 x 100 line: 0.97 ms on 64 blocks, 0.13 ms with eight warps per column.
// ---------------------------------------------------------------------------

// a / b, correctly rounded, for b with the correctly rounded reciprocal y and
// a, b in range: a quotient approximation refined twice by its exact residual
// (P. Markstein, "Computation of elementary functions on the IBM RISC System
// /6000 processor", IBM J. Res. Dev. 34, 1990, theorems 6 and 8: the first
// step is within one ulp, the second rounds correctly).  One reciprocal serves
// every division by the same distance.  In range: b in [2^-20, 2^21], a zero
// or |a| in [2^-102, 2^104], so that no residual or quotient leaves the
// representable numbers.
__device__ __forceinline__ float div_by(float a, float b, float y) {
  float q = __fmul_rn(a, y);
  q = __fmaf_rn(__fmaf_rn(-b, q, a), y, q);
  return __fmaf_rn(__fmaf_rn(-b, q, a), y, q);
}
// 1 / r in double, correctly rounded, for a float r in [2^-100, 2^100]: Newton
// steps from the float reciprocal (relative error 2^-24, 2^-47, then below
// 2^-90 before the last rounding; 1 / r has a 24-bit divisor, so it is at
// least 2^-79 away from a rounding boundary).
__device__ __forceinline__ double drcp_float(float r) {
  const double d = (double)r, y0 = (double)__frcp_rn(r);
  const double y1 = __fma_rn(y0, __fma_rn(-d, y0, 1.0), y0);
  return __fma_rn(y1, __fma_rn(-d, y1, 1.0), y1);
}
// coordinates whose differences are zero or at least 2^-64
__device__ __forceinline__ bool in_range(float v) {
  const float a = fabsf(v);
  return a == 0.0f || (a >= 9.094947e-13f && a <= 1.0995116e12f);  // [2^-40, 2^40]
}
// distances whose ratio's third power div_by reaches: [2^-20, 2^21]
__device__ __forceinline__ bool dist_in_range(float v) {
  return v >= 9.5367432e-7f && v <= 2097152.0f;
}

template <int SPLIT>
__global__ void __launch_bounds__(256)
    k_image_compat(float *__restrict__ img, CompatImageArgs a,
                   const float *__restrict__ dips, const int *__restrict__ ints,
                   const float *__restrict__ geom, int ntr,
                   unsigned long long *npt) {
  constexpr int TX = 8 / SPLIT;
  __shared__ OrderedSmem<SPLIT> sm;
  __shared__ float s_red[8][8];
  __shared__ TileBox s_box;
  __shared__ unsigned long long s_cnt;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int iz0 = blockIdx.x * 32, ixb0 = blockIdx.y * TX;
  const int izi = iz0 + lane, ixb = ixb0 + warp / SPLIT;
  const bool live = izi < a.nzi && ixb < a.nxb;
  const int ixi = ixb + a.ixstart;
  const bool act = live && ixi >= a.tcdp1 && ixi <= a.tcdp2;
  if (tid == 0) s_cnt = 0;

  float tan[4] = {0.f, 0.f, 0.f, 0.f};
  float acc = 0.0f;
  if (live) {
    const size_t k = (size_t)ixi * a.nzi + izi;
#pragma unroll
    for (int j = 0; j < 4; ++j) tan[j] = dips[j * a.nxz + k];
    acc = img[(size_t)ixb * a.nzi + izi];
  }
  // Per-point constants of image_depth_gpu (src/q-psdm.cu:2303-2330).
  const float tz = a.taperzone;
  DipLimits d;
  d.x1 = tan[0], d.x2 = tan[1], d.y1 = tan[2], d.y2 = tan[3];
  d.x1c = __fsub_rn(d.x1, __fmul_rn(tz, __fadd_rn(1.0f, __fmul_rn(d.x1, d.x1))));
  d.x2c = __fadd_rn(d.x2, __fmul_rn(tz, __fadd_rn(1.0f, __fmul_rn(d.x2, d.x2))));
  d.y1c = __fsub_rn(d.y1, __fmul_rn(tz, __fadd_rn(1.0f, __fmul_rn(d.y1, d.y1))));
  d.y2c = __fadd_rn(d.y2, __fmul_rn(tz, __fadd_rn(1.0f, __fmul_rn(d.y2, d.y2))));
  d.wide = d.x1 > d.x1c && d.x2 < d.x2c && d.y1 > d.y1c && d.y2 < d.y2c;
  const float z = __fmul_rn((float)izi, a.dzi);
  const float z2 = __fmul_rn(z, z);
  const float x = __fmul_rn((float)ixi, a.dxi);
  tile_limits(act, d.x1c, d.x2c, d.y1c, d.y2c, s_red);
  // the tile's columns inside the tables, and its rows
  const int col_lo = max(ixb0 + a.ixstart, a.tcdp1);
  const int col_hi = min(min(ixb0 + TX, a.nxb) - 1 + a.ixstart, a.tcdp2);
  const int nrow = min(32, a.nzi - iz0);
  __syncthreads();
  if (tid == 0)
    s_box = tile_box(s_red, col_lo * a.dxi, col_hi * a.dxi, iz0 * a.dzi,
                     (iz0 + nrow - 1) * a.dzi);
  // ts = tg = 1 in the reference: t, the sample indices and v are constants.
  const float t = 2.0f;
  const int it1 = __float2int_rz(__fdiv_rn(t, a.dt1));
  const bool t_ok = it1 > 0 && it1 + 1 < a.nt;
  const float v0 = ((double)t > 0.1) ? __fdiv_rn(100.0f, __fmul_rn(t, t))
                                     : __fmul_rn(100.0f, 100.0f);
  const bool z_ok = in_range(z) && in_range(x);
  unsigned cnt = 0;
  // source terms, reused while consecutive traces share a source
  float last_sx = NAN, last_sy = NAN, ds = 0.f, sax = 0.f, say = 0.f, saz = 0.f;

  auto keep = [&](int i, int4 &r, float4 &g, float2 &h) {
    h = make_float2(0.0f, 0.0f);
    const int4 q0 = *reinterpret_cast<const int4 *>(ints + (size_t)i * kGateInts);
    if (q0.x != kAccepted) return false;
    const int4 q1 = *reinterpret_cast<const int4 *>(ints + (size_t)i * kGateInts + 4);
    const int lo = max(q1.x, col_lo), hi = min(q1.y, col_hi);
    const int rows = iz0 + nrow - max(q1.w, iz0);
    if (lo > hi || rows <= 0) return false;
    cnt += (unsigned)((hi - lo + 1) * rows);  // a point-trace: a pair in the aperture
    g = *reinterpret_cast<const float4 *>(geom + (size_t)i * kGateF);
    const bool ok = in_range(g.x) && in_range(g.y) && in_range(g.z) && in_range(g.w);
    r = make_int4(lo, hi, q1.w, ok);
    return t_ok && tile_keep(make_float2(g.x, g.y), make_float2(g.z, g.w), s_box);
  };
  auto eval = [&](int k, float &val) {
    const int4 r = sm.rec[k];
    const float4 gm = sm.geo[k];
    if (ixi < r.x || ixi > r.y || izi < r.z) return false;
    if (gm.x != last_sx || gm.y != last_sy) {
      last_sx = gm.x;
      last_sy = gm.y;
      const float dsx = __fsub_rn(gm.x, x);
      ds = __fsqrt_rn(__fadd_rn(__fadd_rn(__fmul_rn(dsx, dsx), __fmul_rn(gm.y, gm.y)), z2));
      sax = __fdiv_rn(dsx, ds), say = __fdiv_rn(gm.y, ds), saz = __fdiv_rn(z, ds);
    }
    const float dgx = __fsub_rn(gm.z, x);
    const float dg =
        __fsqrt_rn(__fadd_rn(__fadd_rn(__fmul_rn(dgx, dgx), __fmul_rn(gm.w, gm.w)), z2));
    const float y = __frcp_rn(dg);
    // no quotient leaves div_by's range
    const bool fast = r.w && z_ok && dist_in_range(dg) && dist_in_range(ds);
    auto over_dg = [&](float n) { return fast ? div_by(n, dg, y) : __fdiv_rn(n, dg); };
    const float ux = __fadd_rn(sax, over_dg(dgx));
    const float uy = __fadd_rn(say, over_dg(gm.w));
    const float uz = __fadd_rn(saz, over_dg(z));
    // The reference rejects `tanx <= tanx1c || tanx2c <= tanx || ...`; the
    // negated form agrees for every number and also rejects a NaN tangent
    // (0/0 at z = 0 for collinear source, receiver and node), as the
    // reference binary does: its approximate divisions give +-inf there.
    float w;
    if (!dip_taper(ux, uy, uz, d, w)) return false;
    // tr = ds/dg*ds/dg*ds/dg*tg/ts, evaluated left to right (tg = ts = 1).
    float q = over_dg(ds);
    q = over_dg(__fmul_rn(q, ds));
    q = over_dg(__fmul_rn(q, ds));
    const double rd = (double)q;
    const double ri = q >= 7.9e-31f && q <= 1.26e30f ? drcp_float(q) : __ddiv_rn(1.0, rd);
    q = __double2float_rn(__dmul_rn((double)w, __dadd_rn(rd, ri)));
    val = __fmul_rn(v0, q);
    return true;
  };
  ordered_walk<SPLIT>(sm, ntr, act, keep, eval, [&](float v) { acc = __fadd_rn(acc, v); });
  if (live && (SPLIT == 1 || warp % SPLIT == 0)) img[(size_t)ixb * a.nzi + izi] = acc;
  if (npt) {
    // warp-aggregate the point-trace count
    for (int off = 16; off > 0; off >>= 1) cnt += __shfl_down_sync(0xffffffffu, cnt, off);
    if (lane == 0 && cnt) atomicAdd(&s_cnt, (unsigned long long)cnt);
    __syncthreads();
    if (tid == 0 && s_cnt) atomicAdd(npt, s_cnt);
  }
}

int launch_image_compat(float *d_img, const CompatImageArgs &a,
                        const float *d_dips, const int *d_ints,
                        const float *d_geom, int ntr, unsigned long long *d_npt,
                        cudaStream_t s) {
  if (ntr <= 0) return QPSDM_OK;
  ordered_by_split(a.nzi, a.nxb, 32, [&](auto split) {
    constexpr int S = decltype(split)::value;
    const dim3 grid((a.nzi + 31) / 32, (a.nxb + 8 / S - 1) / (8 / S));
    k_image_compat<S><<<grid, 256, 0, s>>>(d_img, a, d_dips, d_ints, d_geom, ntr, d_npt);
  });
  return cudaGetLastError() == cudaSuccess ? QPSDM_OK : QPSDM_ECUDA;
}

}  // namespace qpsdm

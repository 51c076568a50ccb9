// eikonal.cu -- traveltime and t* tables from a gridded velocity / Q model.
//
// The reference reads precomputed tables (L<line>.ttt / .qqq,
// src/q-psdm.cu:2382-2627); this is the generator that writes them.  Each
// source (a surface node of a table's local grids) gets its own local 3D grid
// (origin ox, oy at the surface, spacing h, common size per batch).  The
// eikonal equation |grad T| = 1/v is solved by first-order Godunov upwind
// updates (the update of Zhao's fast sweeping method, run as in-place
// parallel relaxation: each update only lowers T and stays an upper bound, so
// the iteration reaches the same fixed point as ordered sweeps), started from
// the linear-gradient analytic traveltime inside a radius around the source,
// which is held fixed.  t* then follows from grad T . grad t* = 1/(v^2 Q)
// with the same upwind neighbours:
//   t*_i = (f_i + sum_d w_d t*_d) / sum_d w_d,  w_d = (T_i - T_d)/h^2,
// accumulated in double precision (t* is a cumulative integral along the
// ray; the float result is written once, at the end).
#include <math.h>

#include <algorithm>

#include "common.cuh"
#include "qpsdm_engine.h"

namespace qpsdm {

constexpr float kInf = 1e30f;

// Trilinear sample of a global model grid [nz][ny][nx] (clamped at edges).
__device__ __forceinline__ float model_at(const float *__restrict__ g, const qpsdm_eik_model &m,
                                          float x, float y, float z) {
  const float fx = fminf(fmaxf((x - m.ox) / m.h, 0.0f), (float)(m.nx - 1));
  const float fy = fminf(fmaxf((y - m.oy) / m.h, 0.0f), (float)(m.ny - 1));
  const float fz = fminf(fmaxf(z / m.h, 0.0f), (float)(m.nz - 1));
  const int ix = min((int)fx, max(m.nx - 2, 0)), iy = min((int)fy, max(m.ny - 2, 0));
  const int iz = min((int)fz, max(m.nz - 2, 0));
  const float wx = m.nx > 1 ? fx - ix : 0.f, wy = m.ny > 1 ? fy - iy : 0.f;
  const float wz = m.nz > 1 ? fz - iz : 0.f;
  const size_t sx = m.nx > 1 ? 1 : 0, sy = m.ny > 1 ? (size_t)m.nx : 0;
  const size_t sz = m.nz > 1 ? (size_t)m.nx * m.ny : 0;
  const float *p = g + ((size_t)iz * m.ny + iy) * m.nx + ix;
  const float c00 = p[0] + wx * (p[sx] - p[0]);
  const float c01 = p[sy] + wx * (p[sy + sx] - p[sy]);
  const float c10 = p[sz] + wx * (p[sz + sx] - p[sz]);
  const float c11 = p[sz + sy] + wx * (p[sz + sy + sx] - p[sz + sy]);
  const float c0 = c00 + wy * (c01 - c00), c1 = c10 + wy * (c11 - c10);
  return c0 + wz * (c1 - c0);
}

// Linear-gradient traveltime from a surface point (v = v0 + k z).
__device__ __forceinline__ float lin_grad_time(float r, float z, float v0, float k) {
  if (k < 1e-6f) return sqrtf(r * r + z * z) / v0;
  const float v = v0 + k * z;
  const float arg = 1.0f + k * k * (r * r + z * z) / (2.0f * v0 * v);
  return acoshf(fmaxf(arg, 1.0f)) / k;
}

// A batch of local grids is relaxed in blocks of kEx x kEy x kEz nodes, one CTA
// a block, two nodes a thread.  Only blocks that can change are visited: a
// block whose nodes or facing neighbours changed in a sweep is on the next
// sweep's list (a node's update depends on its six neighbours alone, so a
// node left out would have kept its value).  Lists, the sweep a block was last
// listed for and the marks of blocks with start nodes (the only ones that sweep
// 0 visits; for t*, then, of blocks visited) live in the t* output until it is written.
constexpr int kEx = 16, kEy = 8, kEz = 4, kEikThreads = kEx * kEy * kEz / 2;

// n / d for n < 2^31 as a multiply-high and a shift: with 2^(l-1) < d <= 2^l,
// mul = ceil(2^(31+l) / d) is exact (Granlund and Montgomery, "Division by
// invariant integers using multiplication", 1994).
struct EikDiv {
  unsigned d, mul;
  int shift;  // l - 1; unused for d = 1
  EikDiv() = default;
  explicit EikDiv(unsigned n) : d(n), mul(0), shift(0) {
    int l = 0;
    while ((1ull << l) < n) ++l;
    if (n > 1) mul = (unsigned)(((1ull << (31 + l)) + n - 1) / n), shift = l - 1;
  }
  __device__ __forceinline__ int div(int n) const {
    return d == 1 ? n : (int)(__umulhi((unsigned)n, mul) >> shift);
  }
};

struct EikBlocks {
  qpsdm_eik_grid g;
  int nbx, nby, nbz, nblk;  // blocks per axis, blocks of all sources
  EikDiv row, plane, grid;  // by nbx, nbx nby, nbx nby nbz
  int *list0, *list1;       // blocks of even and odd sweeps, [nblk] each
  int *listed, *seed;       // sweep a block was last listed for; holds start nodes / visited
  unsigned *count;          // list lengths of three consecutive sweeps, in turn
};

struct EikBlock {
  int s, x0, y0, z0;  // source and first node
  size_t base;        // first node's index
};
__device__ __forceinline__ EikBlock eik_block(const EikBlocks &B, int b) {
  EikBlock e;
  e.s = B.grid.div(b);
  int r = b - e.s * (int)B.grid.d;
  const int bz = B.plane.div(r);
  r -= bz * (int)B.plane.d;
  const int by = B.row.div(r);
  e.x0 = (r - by * B.nbx) * kEx;
  e.y0 = by * kEy;
  e.z0 = bz * kEz;
  e.base = (((size_t)e.s * B.g.nz + e.z0) * B.g.ny + e.y0) * B.g.nx + e.x0;
  return e;
}
// Lists block b's neighbours (bit 1 + 2 axis + (upper side)) and itself (bit 0)
// for the next sweep; threads 0 .. 6 of the CTA.
__device__ __forceinline__ void eik_mark(const EikBlocks &B, int b, const EikBlock &e,
                                         unsigned faces, int sweep) {
  const int t = threadIdx.x;
  if (t > 6 || !((faces >> t) & 1u)) return;
  int o = b;
  if (t > 0) {
    const int step = t < 3 ? 1 : t < 5 ? B.nbx : B.nbx * B.nby;
    const int at = t < 3 ? e.x0 / kEx : t < 5 ? e.y0 / kEy : e.z0 / kEz;
    const bool up = !(t & 1);
    if (up ? at + 1 >= (t < 3 ? B.nbx : t < 5 ? B.nby : B.nbz) : at == 0) return;
    o += up ? step : -step;
  }
  if (atomicExch(B.listed + o, sweep + 1) == sweep + 1) return;
  (sweep & 1 ? B.list0 : B.list1)[atomicAdd(B.count + (sweep + 1) % 3, 1u)] = o;
}
// Which faces of its block a changed node lies on, and the block itself.
__device__ __forceinline__ unsigned eik_faces(int lx, int ly, int lz) {
  return 1u | (lx == 0 ? 2u : 0u) | (lx == kEx - 1 ? 4u : 0u) | (ly == 0 ? 8u : 0u) |
         (ly == kEy - 1 ? 16u : 0u) | (lz == 0 ? 32u : 0u) | (lz == kEz - 1 ? 64u : 0u);
}

// Per node: h/v (negative: a start node, held at its analytic value) and
// 1/(v^2 Q), and the start values near the source.
__global__ void k_eik_setup(const float *__restrict__ vel, const float *__restrict__ invq,
                            qpsdm_eik_model m, const float4 *__restrict__ src, EikBlocks B,
                            float r0, float *__restrict__ F, float *__restrict__ QF,
                            float *__restrict__ T, double *__restrict__ TS) {
  const qpsdm_eik_grid g = B.g;
  if (blockIdx.x == 0 && threadIdx.x < 3) B.count[threadIdx.x] = 0;
  for (int b = blockIdx.x; b < B.nblk; b += gridDim.x) {
    const EikBlock e = eik_block(B, b);
    bool start = false;
    const float4 sp = src[e.s];  // source x, y; local grid origin ox, oy
    const float qs = model_at(invq, m, sp.x, sp.y, 0.0f);  // near-surface Q on the path
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int l = threadIdx.x + h * kEikThreads;
      const int lx = l % kEx, ly = l / kEx % kEy, lz = l / (kEx * kEy);
      if (e.x0 + lx >= g.nx || e.y0 + ly >= g.ny || e.z0 + lz >= g.nz) continue;
      const size_t i = e.base + ((size_t)lz * g.ny + ly) * g.nx + lx;
      const float x = sp.z + (e.x0 + lx) * g.h, y = sp.w + (e.y0 + ly) * g.h;
      const float z = (e.z0 + lz) * g.h;
      const float v = fmaxf(model_at(vel, m, x, y, z), 1.0f);
      QF[i] = model_at(invq, m, x, y, z) / (v * v);
      const float dx = x - sp.x, dy = y - sp.y;
      if (dx * dx + dy * dy + z * z <= r0 * r0) {
        const float t = lin_grad_time(sqrtf(dx * dx + dy * dy), z, m.v0, m.kz);
        F[i] = -(g.h / v);
        T[i] = t;
        TS[i] = (double)t * qs;
        start = true;
      } else {
        F[i] = g.h / v;
        T[i] = kInf;
        TS[i] = 0.0;
      }
    }
    start = __syncthreads_or(start);
    if (threadIdx.x == 0) {
      B.listed[b] = -1;
      B.seed[b] = start;
    }
  }
}

// Godunov update of a node from the smaller neighbour value of each axis.
__device__ __forceinline__ float eik_update(float a, float b, float c, float f) {
  const float t0 = fminf(a, fminf(b, c)), t2 = fmaxf(a, fmaxf(b, c));
  const float t1 = fminf(fmaxf(a, b), fmaxf(fminf(a, b), c));  // middle value
  if (t0 >= kInf) return kInf;
  float t = t0 + f;
  if (t > t1 && t1 < kInf) {
    const float s2 = t0 + t1, d2 = 2.0f * f * f - (t0 - t1) * (t0 - t1);
    t = 0.5f * (s2 + sqrtf(fmaxf(d2, 0.0f)));
    if (t > t2 && t2 < kInf) {
      const float s3 = t0 + t1 + t2;
      const float d3 = s3 * s3 - 3.0f * (t0 * t0 + t1 * t1 + t2 * t2 - f * f);
      t = (s3 + sqrtf(fmaxf(d3, 0.0f))) / 3.0f;
    }
  }
  return t;
}

// Godunov relaxation of the listed blocks (sweep 0: those with start nodes),
// each with its halo in shared memory, red nodes and black nodes in turn (a
// node's neighbours are all of the other colour: no node is read while it is
// written), until
// nothing changes, kEikInner times at most.  A thread has one node of each
// colour, neighbours in x.  Rows of 24 words: a warp's 8 x 4 nodes of one
// colour lie in 32 banks.
//
// Bound by issue, and by the colours taking turns at a barrier.  28 M nodes, 32
// sources: 256 sweeps over every node, in global memory, took 70 ms; over listed
// blocks, one update a visit, 15.4 ms in 224 sweeps; now 5.4 ms in 80.  With 1,
// 2, 4, 8, 16 updates a visit at most, and 7 ms of t* in each: 26.5, 20.8, 14.9,
// 13.1, 12.9 ms.
//
// The price is in T's rounding.  The FP32 update rounds by some eps T^2 / f, a
// node keeps the lowest of its values, and the order of updates decides how far
// below the fixed point it creeps: T's error against 64 bits, relative 2e-5 to
// 5e-4, is 1.2 times the full sweeps' (geometric mean of 64 models, 3 to 8 sources
// each; 0.9 to 1.6 in most, 2.7 where the full sweeps' was 1.6e-5), t*'s 1.03 to
// 1.09 times.  One update a visit from global memory had 1.03 times (1.26 at
// most) in 23 ms, ignoring changes below 1e-6 of T instead of 1e-7 1.0 times (2.1)
// in this kernel's time.  Neither was taken: t* takes its upwind neighbours by T,
// so with any other T near ties fall the other way, and results would leave this
// solver's by some 1e-4 of t*, more than FP32 rounding accounts for.
constexpr int kEikInner = 8;
__global__ void __launch_bounds__(kEikThreads)
    k_eik_relax(const float *__restrict__ F, float *__restrict__ T, EikBlocks B, int sweep) {
  constexpr int HX = 24, HY = kEy + 2, HZ = kEz + 2;
  __shared__ float s_t[HX * HY * HZ];
  __shared__ unsigned s_faces;
  const qpsdm_eik_grid g = B.g;
  const size_t sxy = (size_t)g.nx * g.ny;
  const int n = sweep == 0 ? B.nblk : (int)B.count[sweep % 3];
  if (blockIdx.x == 0 && threadIdx.x == 0) B.count[(sweep + 2) % 3] = 0;
  const int tid = threadIdx.x;
  const int px = tid % (kEx / 2), ly = tid / (kEx / 2) % kEy, lz = tid / (kEx / 2 * kEy);
  const int odd = (ly + lz) & 1;
  // node c (0 red, 1 black) of this thread
  const int lx[2] = {2 * px + odd, 2 * px + (odd ^ 1)};
  const int row = ((lz + 1) * HY + ly + 1) * HX + 1;
  for (int k = blockIdx.x; k < n; k += gridDim.x) {
    if (sweep == 0 && !B.seed[k]) continue;  // uniform in the CTA
    const int blk = sweep == 0 ? k : (sweep & 1 ? B.list1 : B.list0)[k];
    const EikBlock e = eik_block(B, blk);
    if (tid == 0) s_faces = 0;
    const bool in_yz = e.y0 + ly < g.ny && e.z0 + lz < g.nz;
    const size_t i0 = e.base + lz * sxy + (size_t)ly * g.nx;
    float f[2], t[2], old[2];
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const bool in = in_yz && e.x0 + lx[c] < g.nx;
      f[c] = in ? F[i0 + lx[c]] : -kInf;
      old[c] = t[c] = in ? T[i0 + lx[c]] : kInf;
      s_t[row + lx[c]] = t[c];
    }
    // halo: z faces (two rows of 128), y faces (64 each), x faces (32 each)
    auto halo = [&](int hx, int hy, int hz) {
      const int x = e.x0 + hx, y = e.y0 + hy, z = e.z0 + hz;
      const bool in = x >= 0 && x < g.nx && y >= 0 && y < g.ny && z >= 0 && z < g.nz;
      s_t[((hz + 1) * HY + hy + 1) * HX + hx + 1] =
          in ? T[e.base + hz * (ptrdiff_t)sxy + hy * (ptrdiff_t)g.nx + hx] : kInf;
    };
    halo(tid % kEx, tid / kEx % kEy, tid < 128 ? -1 : kEz);
    if (tid < 128)
      halo(tid % kEx, tid < 64 ? -1 : kEy, tid / kEx % kEz);
    else if (tid < 192)
      halo(tid < 160 ? -1 : kEx, tid % kEy, tid / kEy % kEz);
    __syncthreads();
    bool more = true;
    for (int it = 0; it < kEikInner && more; ++it) {
      bool ch = false;
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        if (f[c] >= 0.0f) {
          const float *p = s_t + row + lx[c];
          const float v = eik_update(fminf(p[-1], p[1]), fminf(p[-HX], p[HX]),
                                     fminf(p[-HX * HY], p[HX * HY]), f[c]);
          if (v < t[c] * (1.0f - 1e-7f)) {
            t[c] = v;
            s_t[row + lx[c]] = v;
            ch = true;
          }
        }
        if (c == 0) __syncthreads();
      }
      more = __syncthreads_or(ch);
    }
    unsigned faces = 0;
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      if (t[c] < old[c]) T[i0 + lx[c]] = t[c];
      // (sweep 0 lists what start nodes reach)
      if (t[c] < old[c] || (sweep == 0 && f[c] < 0.0f && f[c] > -kInf))
        faces |= eik_faces(lx[c], ly, lz) & ~1u;
    }
    if (more) faces |= 1u;  // settled, unless the loop ran out
    if (faces) atomicOr(&s_faces, faces);
    __syncthreads();
    eik_mark(B, blk, e, s_faces, sweep);
    __syncthreads();  // s_faces is cleared for the next block
  }
}

// t* of the listed blocks along the upwind directions of T (FP64), one node a
// thread: a block with its halo in shared memory is relaxed until nothing in
// it changes.  In sweep 0 the blocks that hold start nodes, and after it what
// they reach: t* at a node depends on nodes of smaller T only, so the values
// settle outwards from the source, most blocks in a few visits, and a block is
// listed only for a neighbour of smaller T that has changed, or whose block is
// visited for the first time: a value that stays at its initial 0 (no attenuation
// so far) must be carried on too.  256 sweeps over every
// node took 95 ms for the 28 M nodes of 32 sources; so 6.9 ms; 4.7 ms with the
// traveltimes of the neighbours from shared memory, a halo of the facing nodes
// only and the seed marks (a visit's preparation, not its FP64 updates, is most
// of its instructions: three updates to a barrier gave nothing).
constexpr int kTsThreads = kEx * kEy * kEz;
__global__ void __launch_bounds__(kTsThreads)
    k_tstar_relax(const float *__restrict__ F, const float *__restrict__ T,
                  const float *__restrict__ QF, double *__restrict__ TS, EikBlocks B, int sweep) {
  constexpr int HX = kEx + 2, HY = kEy + 2, HZ = kEz + 2;
  __shared__ double s_ts[HX * HY * HZ];
  __shared__ float s_t[HX * HY * HZ];
  __shared__ unsigned s_faces;
  const qpsdm_eik_grid g = B.g;
  const size_t sxy = (size_t)g.nx * g.ny;
  const double ih2 = 1.0 / ((double)g.h * g.h);
  const int n = sweep == 0 ? B.nblk : (int)B.count[sweep % 3];
  if (blockIdx.x == 0 && threadIdx.x == 0) B.count[(sweep + 2) % 3] = 0;
  const int lx = threadIdx.x % kEx, ly = threadIdx.x / kEx % kEy, lz = threadIdx.x / (kEx * kEy);
  const int at = ((lz + 1) * HY + ly + 1) * HX + lx + 1;
  // this thread's node of the halo: z faces (128 each), y faces (64 each), x faces (32 each)
  const int u = threadIdx.x;
  int hx = -2, hy = 0, hz = 0;
  if (u < 256)
    hx = u % kEx, hy = u / kEx % kEy, hz = u < 128 ? -1 : kEz;
  else if (u < 384)
    hx = u % kEx, hy = u < 320 ? -1 : kEy, hz = u / kEx % kEz;
  else if (u < 448)
    hx = u < 416 ? -1 : kEx, hy = u % kEy, hz = u / kEy % kEz;
  for (int k = blockIdx.x; k < n; k += gridDim.x) {
    if (sweep == 0 && !B.seed[k]) continue;  // uniform in the CTA
    const int blk = sweep == 0 ? k : (sweep & 1 ? B.list1 : B.list0)[k];
    const EikBlock e = eik_block(B, blk);
    bool on = e.x0 + lx < g.nx && e.y0 + ly < g.ny && e.z0 + lz < g.nz;
    const size_t i = e.base + lz * sxy + (size_t)ly * g.nx + lx;
    const bool start = on && F[i] < 0.0f;
    const bool first = sweep == 0 || !B.seed[blk];  // seed: blocks visited, from here on
    if (threadIdx.x == 0) s_faces = 0;
    // the block and the nodes facing it
    const float ti = on ? T[i] : kInf;
    const double old = on ? TS[i] : 0.0;
    s_t[at] = ti;
    s_ts[at] = old;
    if (hx > -2) {
      const int x = e.x0 + hx, y = e.y0 + hy, z = e.z0 + hz;
      const bool in = x >= 0 && x < g.nx && y >= 0 && y < g.ny && z >= 0 && z < g.nz;
      const ptrdiff_t o = hz * (ptrdiff_t)sxy + hy * (ptrdiff_t)g.nx + hx;
      const int j = ((hz + 1) * HY + hy + 1) * HX + hx + 1;
      s_t[j] = in ? T[e.base + o] : kInf;
      s_ts[j] = in ? TS[e.base + o] : 0.0;
    }
    __syncthreads();
    // the update's terms: upwind neighbours and weights
    int nb[3] = {at, at, at};
    double w[3] = {0.0, 0.0, 0.0}, q = 0.0, rden = 0.0, val = old;
    unsigned faces = 0;  // sides whose outside neighbour lies downwind
    if (on) {
      const int hd[3] = {1, HX, HX * HY};
      double den = 0.0;
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        const float lo = s_t[at - hd[d]], hi = s_t[at + hd[d]];
        const float best = fminf(lo, hi);
        if (best < ti) {
          w[d] = ((double)ti - (double)best) * ih2;
          nb[d] = at + (lo <= hi ? -hd[d] : hd[d]);
          den += w[d];
        }
        faces |= (lo > ti ? 2u : 0u) << (2 * d) | (hi > ti ? 4u : 0u) << (2 * d);
      }
      faces &= eik_faces(lx, ly, lz);
      on = !start && ti < kInf && den > 0.0;
      if (on) {
        rden = 1.0 / den;
        q = QF[i];
      }
    }
    bool more = true;
    for (int it = 0; it < 64 && more; ++it) {
      bool ch = false;
      if (on) {
        double num = q;
#pragma unroll
        for (int d = 0; d < 3; ++d) num += w[d] * s_ts[nb[d]];
        const double v = num * rden;
        // (bits: a NaN settles too)
        ch = __double_as_longlong(v) != __double_as_longlong(val);
        if (ch) s_ts[at] = val = v;
      }
      more = __syncthreads_or(ch);
    }
    if (on && __double_as_longlong(val) != __double_as_longlong(old))
      TS[i] = val;
    else if (!first)
      faces = 0;
    if (more) faces |= 1u;  // settled, unless the loop ran out
    if (faces) atomicOr(&s_faces, faces);
    if (threadIdx.x == 0) B.seed[blk] = 1;
    __syncthreads();
    eik_mark(B, blk, e, s_faces, sweep);
    __syncthreads();
  }
}

__global__ void k_tstar_store(const double *__restrict__ TS, float *__restrict__ out, size_t n) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x)
    out[i] = (float)TS[i];
}

// Table entries (reference layout) whose source is solved in this batch.
// Entry e of the table (cells in descriptor order, cell_base prefix sums of
// block sizes) = cell c, surface node, ixl, izl; node_src gives the global
// source number of every (cell, node) (node_base prefix sums per cell).
__global__ void k_eik_fill(const float *__restrict__ T, const float *__restrict__ TS,
                           qpsdm_eik_grid g, const float4 *__restrict__ src, int s0, int ns,
                           const qpsdm_ttt_desc *__restrict__ desc,
                           const int64_t *__restrict__ cell_base, const int *__restrict__ node_base,
                           const int *__restrict__ node_src, int ncell, qpsdm_eik_fill_geom fg,
                           float *__restrict__ ttt, float *__restrict__ qqq) {
  const int64_t total = cell_base[ncell];
  const size_t n = (size_t)g.nx * g.ny * g.nz;
  const int per_node = fg.nxi1 * fg.nzi1;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total;
       e += (int64_t)gridDim.x * blockDim.x) {
    int lo = 0, hi = ncell;
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (cell_base[mid] <= e) lo = mid; else hi = mid;
    }
    const int c = lo;
    const int64_t r = e - cell_base[c];
    const int node = (int)(r / per_node);
    const int rem = (int)(r - (int64_t)node * per_node);
    const int ixl = rem / fg.nzi1, izl = rem - ixl * fg.nzi1;
    const int sl = node_src[node_base[c] + node] - s0;
    if (sl < 0 || sl >= ns) continue;
    const float4 sp = src[sl];
    const int ixg = c / fg.nzg, izg = c - ixg * fg.nzg;
    const float x = fg.x_cdp1 + (ixg * fg.nxi1 + ixl) * fg.dxi;
    const float z = (izg * fg.nzi1 + izl) * fg.dzii;
    const float fx = fminf(fmaxf((x - sp.z) / g.h, 0.0f), (float)(g.nx - 1) - 1e-3f);
    const float fy = fminf(fmaxf((fg.line_y - sp.w) / g.h, 0.0f), (float)(g.ny - 1) - 1e-3f);
    const float fz = fminf(fmaxf(z / g.h, 0.0f), (float)(g.nz - 1) - 1e-3f);
    const int jx = (int)fx, jy = (int)fy, jz = (int)fz;
    const float wx = fx - jx, wy = fy - jy, wz = fz - jz;
    const size_t base = (size_t)sl * n + ((size_t)jz * g.ny + jy) * g.nx + jx;
    const size_t sx = 1, sy = g.ny > 1 ? (size_t)g.nx : 0, sz = (size_t)g.nx * g.ny;
    float out[2];
    const float *arr[2] = {T, TS};
#pragma unroll
    for (int w = 0; w < 2; ++w) {
      const float *p = arr[w] + base;
      const float c00 = p[0] + wx * (p[sx] - p[0]);
      const float c01 = p[sy] + wx * (p[sy + sx] - p[sy]);
      const float c10 = p[sz] + wx * (p[sz + sx] - p[sz]);
      const float c11 = p[sz + sy] + wx * (p[sz + sy + sx] - p[sz + sy]);
      const float c0 = c00 + wy * (c01 - c00), c1 = c10 + wy * (c11 - c10);
      out[w] = c0 + wz * (c1 - c0);
    }
    ttt[desc[c].idx + r] = out[0];
    qqq[desc[c].idx + r] = out[1];
  }
}

}  // namespace qpsdm

using namespace qpsdm;

extern "C" int qpsdm_eikonal_solve(const float *d_vel, const float *d_invq,
                                   const qpsdm_eik_model *model, const float *d_src, int nsrc,
                                   const qpsdm_eik_grid *grid, float init_radius, int max_iter,
                                   float *d_work, float *d_T, float *d_tstar, void *stream) {
  if (!d_vel || !d_invq || !model || !d_src || !grid || !d_work || !d_T || !d_tstar ||
      nsrc <= 0 || grid->nx < 2 || grid->ny < 1 || grid->nz < 2 || grid->h <= 0.f ||
      model->nx < 1 || model->ny < 1 || model->nz < 1 || model->h <= 0.f || max_iter <= 0)
    return QPSDM_EINVAL;
  cudaStream_t st = (cudaStream_t)stream;
  const qpsdm_eik_grid g = *grid;
  const size_t n = (size_t)g.nx * g.ny * g.nz * nsrc;
  // work: F, QF (n floats each), t* in FP64 (n doubles, 8-byte aligned), counts
  float *F = d_work, *QF = d_work + n;
  double *TS = reinterpret_cast<double *>(d_work + 2 * n + ((2 * n) & 1));
  if (reinterpret_cast<uintptr_t>(d_work) % 8) return QPSDM_EINVAL;
  EikBlocks B;
  B.g = g;
  B.nbx = (g.nx + kEx - 1) / kEx;
  B.nby = (g.ny + kEy - 1) / kEy;
  B.nbz = (g.nz + kEz - 1) / kEz;
  const int64_t nblk = (int64_t)nsrc * B.nbx * B.nby * B.nbz;
  if (nblk > 0x7fffffff) return QPSDM_EINVAL;
  B.nblk = (int)nblk;
  B.row = EikDiv(B.nbx);
  B.plane = EikDiv(B.nbx * B.nby);
  B.grid = EikDiv(B.nbx * B.nby * B.nbz);
  // at least four nodes to a block (2, 1, 2 an axis: nx, nz >= 2), so four words
  // per block fit the output
  B.list0 = reinterpret_cast<int *>(d_tstar);
  B.list1 = B.list0 + nblk;
  B.listed = B.list1 + nblk;
  B.seed = B.listed + nblk;
  B.count = reinterpret_cast<unsigned *>(TS + n);
  const float4 *src = (const float4 *)d_src;
  const int grd = (int)std::min<int64_t>(nblk, 148 * 8);
  k_eik_setup<<<grd, kEikThreads, 0, st>>>(d_vel, d_invq, *model, src, B, init_radius, F, QF, d_T,
                                           TS);
  // sweeps in rounds of 16 until no block is listed (or max_iter)
  auto relax = [&](int limit, auto sweep_fn) {
    for (int it = 0; it < limit; it += 16) {
      for (int k = 0; k < 16; ++k) sweep_fn(it + k);
      unsigned left = 0;
      if (cudaMemcpyAsync(&left, B.count + (it + 16) % 3, sizeof(left), cudaMemcpyDeviceToHost,
                          st) != cudaSuccess ||
          cudaStreamSynchronize(st) != cudaSuccess)
        return (int)QPSDM_ECUDA;
      if (!left) break;
    }
    return (int)QPSDM_OK;
  };
  int rc = relax(max_iter, [&](int sweep) {
    k_eik_relax<<<grd, kEikThreads, 0, st>>>(F, d_T, B, sweep);
  });
  if (rc) return rc;
  cudaMemsetAsync(B.count, 0, 3 * sizeof(unsigned), st);
  cudaMemsetAsync(B.listed, 0xff, sizeof(int) * (size_t)nblk, st);
  rc = relax(4 * (g.nx + g.ny + g.nz), [&](int sweep) {
    k_tstar_relax<<<grd, kTsThreads, 0, st>>>(F, d_T, QF, TS, B, sweep);
  });
  if (rc) return rc;
  k_tstar_store<<<148 * 8, 256, 0, st>>>(TS, d_tstar, n);
  return cudaGetLastError() == cudaSuccess ? QPSDM_OK : QPSDM_ECUDA;
}

extern "C" int qpsdm_eikonal_fill(const float *d_T, const float *d_tstar,
                                  const qpsdm_eik_grid *grid, const float *d_src, int s0, int ns,
                                  const qpsdm_ttt_desc *d_desc, const int64_t *d_cell_base,
                                  const int *d_node_base, const int *d_node_src, int ncell,
                                  const qpsdm_eik_fill_geom *fg, float *d_ttt, float *d_qqq,
                                  void *stream) {
  if (!d_T || !d_tstar || !grid || !d_src || !d_desc || !d_cell_base || !d_node_base ||
      !d_node_src || !fg || !d_ttt || !d_qqq || ncell <= 0 || ns <= 0)
    return QPSDM_EINVAL;
  k_eik_fill<<<148 * 8, 256, 0, (cudaStream_t)stream>>>(
      d_T, d_tstar, *grid, (const float4 *)d_src, s0, ns, d_desc, d_cell_base, d_node_base,
      d_node_src, ncell, *fg, d_ttt, d_qqq);
  return cudaGetLastError() == cudaSuccess ? QPSDM_OK : QPSDM_ECUDA;
}

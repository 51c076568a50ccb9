// physics.cu -- Q-compensated imaging (physics mode) on sm_100a.
//
// The reference's kernel stages per-trace spectra, Q, nf3, the gain-limit
// constants and the ttt/qqq tables (src/q-psdm.cu:2246-2300) but stubs the
// imaging itself (ts = tg = 1, :2350-2351).  This mode computes what those
// inputs describe:
//
//   panels   per accepted trace: t^2 gain + end tapers (as psdm_kernel,
//            :2176-2183), r2c of length nfft, the -i*w band ramp ww of
//            qpsdm() (:1207-1250), the inverse-Q filter
//            A(pi f t*) exp(-2 i f t* ln(f/fc)) with the gain-limit law of
//            lnG/coef1..4 (:1277-1283) for nbins t* values, then c2r of length
//            nffti (the resampled grid dt1, :1201-1206).  The filter table is
//            evaluated once per engine on the host in double precision.
//   image    per image point and trace: traveltime and t* from the tables
//            (bilinear in surface position, linear in depth), t = ts + tg,
//            t* = t*s + t*g, linear interpolation in time and between the two
//            nearest t* panels, the reference's amplitude and dip weights
//            (:2303-2378), accumulated in FP32 (optionally Kahan).
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <math.h>

#include <algorithm>
#include <cstring>
#include <map>
#include <mutex>
#include <tuple>
#include <type_traits>
#include <cmath>
#include <cub/cub.cuh>
#include <vector>

#include "common.cuh"
#include "f32x2.cuh"
#include "fft.cuh"
#include "internal.h"
#include "ordered.cuh"
#include "physics.h"
#include "tile.cuh"

namespace qpsdm {

// One set of the batched form's grouping buffers (receiver keys, members,
// source positions, tile queue, deferred-tile list).  Consecutive image lines
// of a brick alternate between two sets, so that a line's grouping and image
// kernels can run on a second stream beside the previous line's: the tail of
// one line's persistent launch overlaps the start of the next.
struct GroupSet {
  unsigned long long *d_key[2] = {};
  int *d_val[2] = {};
  unsigned long long *d_ukey = nullptr;
  int *d_count = nullptr, *d_off = nullptr, *d_nruns = nullptr;
  int *d_srcflag = nullptr, *d_sid = nullptr;
  float2 *d_srcpos = nullptr;
  int4 *d_mem = nullptr;
  float2 *d_grppos = nullptr;
  int *d_memgrp = nullptr;
  // queue counter, deferred-tile count, finished parts of every tile
  int *d_tile_ctr = nullptr;
  size_t ctr_cap = 0;
  int *d_ndefer = nullptr;  // d_tile_ctr + 1
  int *d_defer = nullptr;
  size_t defer_cap = 0;
  float *d_part = nullptr;  // sums of a split image's member parts
  size_t part_cap = 0;
  int *d_nmem = nullptr;
  void *d_cub = nullptr;
};
// Most parts a tile's members are split into, members of a part's chunks at
// most, and the most sums that the parts of an image leave (32 MB per set, 64
// with compensated sums).
constexpr int kMaxSplit = 32, kSplitChunk = 256;
constexpr size_t kSplitSums = 1 << 23;
constexpr size_t kTabTmpKeep = 1 << 25;  // floats of table staging the plain form keeps

struct PhysicsState {
  int nfft = 0, nffti = 0, nbins = 0, max_batch = 0, dtype = 0;
  float dtstar = 0.0f;
  float4 *d_filter = nullptr;  // [(nbins+1)/2][kmax]: (re, re, im, im) of two bins
  int kmax = 0;                // first frequency bin past the band
  float2 *d_spec = nullptr;    // [max_batch][nfft/2+1]
  float *d_fmax = nullptr;     // [nfft/2+1] max over bins of |filter|
  float *d_pscale = nullptr;   // [max_batch] FP16 panels: per-trace sample multiplier
  void *d_panels = nullptr;    // [max_batch][nbins][nffti]
  float *d_comp = nullptr;     // Kahan compensation, [img_cap]
  size_t comp_cap = 0;
  // line tables
  struct LineTab {
    qpsdm_ttt_desc *dt = nullptr, *dq = nullptr;
    float *ttt = nullptr, *qqq = nullptr;
    size_t dt_cap = 0, dq_cap = 0, ttt_cap = 0, qqq_cap = 0;
    // t and t* tables with identical descriptors: (t, t*) of a node and of the
    // node below it
    float4 *tq = nullptr;
    size_t tq_cap = 0;
    bool paired = false;
    bool one_grid = false;  // every cell has the same surface grid
  };
  std::vector<LineTab> tabs;  // one per line of the brick
  float *d_tab_tmp = nullptr;  // a table from the host before its re-layout
  size_t tab_tmp_cap = 0;
  int ntabs = 0;
  int *d_any = nullptr;       // [max_batch] accepted by any line of the brick
  // batched form: grouping scratch (sized for max_batch at create)
  int form = QPSDM_FORM_PLAIN;
  unsigned long long *d_key[2] = {};  // receiver keys, unsorted / sorted
  int *d_val[2] = {};                 // trace indices, unsorted / sorted
  unsigned long long *d_ukey = nullptr;
  int *d_count = nullptr, *d_off = nullptr, *d_nruns = nullptr;
  int *d_srcflag = nullptr, *d_sid = nullptr;  // source run flags / ids (1-based)
  float2 *d_srcpos = nullptr;                  // [max_batch] source positions
  int4 *d_mem = nullptr;                       // [max_batch] member info
  float2 *d_grppos = nullptr;                  // [max_batch] receiver positions
  int *d_memgrp = nullptr;                     // [max_batch] group of each sorted member
  int *d_tile_ctr = nullptr;
  int *d_defer = nullptr;    // tiles the fast form leaves to k_image_batched
  size_t defer_cap = 0;
  int *d_ndefer = nullptr;
  float *d_part = nullptr;
  size_t part_cap = 0;
  size_t part_words = 1;                       // 2 with compensated sums
  int *d_nmem = nullptr;                       // accepted members of the current line's batch
  void *d_cub = nullptr;
  size_t cub_bytes = 0;
  int num_sms = 0;
  int tile_z = 0, tile_x = 0, forced_variant = 0;
  int variant = -1;          // batched kernel variant (autotuned)
  float *d_tune = nullptr;   // scratch image of the autotuner
  size_t tune_cap = 0;
  float tune_ms[32] = {};    // autotuner timings per variant (ms)
  // the two grouping sets (the d_key .. d_cub fields above are the selected
  // one) and the second stream of the line loop
  GroupSet sets[2];
  int cur_set = 0;
  cudaStream_t aux = nullptr;
  cudaEvent_t ev_fork = nullptr, ev_join = nullptr;
};

// Points the grouping fields at set i (the launches enqueued afterwards use it).
static void select_set(PhysicsState *s, int i) {
  const GroupSet &g = s->sets[i];
  for (int k = 0; k < 2; ++k) {
    s->d_key[k] = g.d_key[k];
    s->d_val[k] = g.d_val[k];
  }
  s->d_ukey = g.d_ukey;
  s->d_count = g.d_count;
  s->d_off = g.d_off;
  s->d_nruns = g.d_nruns;
  s->d_srcflag = g.d_srcflag;
  s->d_sid = g.d_sid;
  s->d_srcpos = g.d_srcpos;
  s->d_mem = g.d_mem;
  s->d_grppos = g.d_grppos;
  s->d_memgrp = g.d_memgrp;
  s->d_tile_ctr = g.d_tile_ctr;
  s->d_defer = g.d_defer;
  s->defer_cap = g.defer_cap;
  s->d_ndefer = g.d_ndefer;
  s->d_part = g.d_part;
  s->part_cap = g.part_cap;
  s->d_nmem = g.d_nmem;
  s->d_cub = g.d_cub;
  s->cur_set = i;
}

static size_t dtype_bytes(int t) { return t == QPSDM_PANEL_FP32 ? 4 : 2; }
static int batched_alloc(PhysicsState *s, const qpsdm_static_params &p);

// (-i ww_k) * A(pi f t*) * exp(-2 i f t* ln(f/fc)) / nfft for every bin, and
// the first frequency bin past the band.
static void filter_table(const qpsdm_static_params &p, int nbins, float dtstar,
                         std::vector<float2> &out, std::vector<float> &fmax, int *kmax) {
  const int nk = p.nfft / 2 + 1;
  const double df = 1.0 / ((double)p.nfft * (double)p.dt);
  const double dw = 2.0 * M_PI * df;
  const int n3 = (int)(p.f3 / df + 0.5), n4 = (int)(p.f4 / df + 0.5);
  const double G = p.threshold, lnG = std::log(G);
  const double c1 = G * (1.0 - lnG - 2.5 * lnG * lnG), c2 = G * (1.0 + 5.0 * lnG);
  const double c3 = -2.5 * G, c4 = 1.1 * G;
  out.assign((size_t)nbins * nk, make_float2(0.f, 0.f));
  *kmax = std::max(1, std::min(nk, std::max(n3, n4)));  // (f3 > f4: a sharp edge at f3)
  for (int b = 0; b < nbins; ++b) {
    const double ts = b * (double)dtstar;
    for (int k = 1; k < nk; ++k) {
      double ww;
      if (k < n3)
        ww = k * dw;
      else if (k < n4)
        ww = n3 * dw * std::pow(std::cos((double)(k - n3) / (n4 - n3) * M_PI * 0.5), 2);
      else
        ww = 0.0;
      const double f = k * df;
      const double x = M_PI * f * ts;
      double a;
      if (x <= lnG)
        a = std::exp(x);
      else if (x <= lnG + 0.2)
        a = c1 + c2 * x + c3 * x * x;
      else
        a = c4;
      const double ph = -2.0 * f * ts * std::log(f / p.fc);
      // (-i ww) * a * (cos ph + i sin ph) / nfft
      const double re = ww * a * std::sin(ph) / p.nfft;
      const double im = -ww * a * std::cos(ph) / p.nfft;
      out[(size_t)b * nk + k] = make_float2((float)re, (float)im);
    }
  }
  fmax.assign(nk, 0.0f);
  for (int b = 0; b < nbins; ++b)
    for (int k = 0; k < nk; ++k) {
      const float2 v = out[(size_t)b * nk + k];
      fmax[k] = std::max(fmax[k], std::hypot(v.x, v.y) * 1.0001f);
    }
}

int physics_create(PhysicsState **out, const qpsdm_static_params &p, std::string *err) {
  *out = nullptr;
  if (p.nbins < 2 || p.nbins > 256 || p.dtstar <= 0.0f) {
    if (err) *err = "physics mode needs 2 <= nbins <= 256 and dtstar > 0";
    return QPSDM_EINVAL;
  }
  if (p.panel_dtype < 0 || p.panel_dtype > 2) {
    if (err) *err = "bad panel dtype";
    return QPSDM_EINVAL;
  }
  if (p.form == QPSDM_FORM_BATCHED && p.max_batch >= (1 << 24)) {
    if (err) *err = "batched form: max_batch must be below 2^24 traces";
    return QPSDM_EINVAL;
  }
  auto *s = new PhysicsState;
  s->nfft = p.nfft;
  s->nffti = p.nffti;
  s->nbins = p.nbins;
  s->dtstar = p.dtstar;
  s->max_batch = p.max_batch;
  s->dtype = p.panel_dtype;
  s->part_words = p.kahan ? 2 : 1;
  std::vector<float2> f;
  std::vector<float> fmax;
  filter_table(p, p.nbins, p.dtstar, f, fmax, &s->kmax);
  const size_t nk = (size_t)p.nfft / 2 + 1;
  auto bad = [&](const char *w) {
    if (err) *err = std::string("physics_create: ") + w;
    physics_destroy(s);
    return QPSDM_ENOMEM;
  };
  std::vector<float4> pairs((size_t)(p.nbins + 1) / 2 * s->kmax, make_float4(0.f, 0.f, 0.f, 0.f));
  for (int q = 0; q < p.nbins; ++q)
    for (int k = 0; k < s->kmax; ++k) {
      float *d = &pairs[(size_t)(q / 2) * s->kmax + k].x;
      d[q & 1] = f[q * nk + k].x;
      d[2 + (q & 1)] = f[q * nk + k].y;
    }
  if (cudaMalloc(&s->d_filter, sizeof(float4) * pairs.size()) != cudaSuccess) return bad("filter");
  cudaMemcpy(s->d_filter, pairs.data(), sizeof(float4) * pairs.size(), cudaMemcpyHostToDevice);
  if (cudaMalloc(&s->d_spec, sizeof(float2) * nk * p.max_batch) != cudaSuccess) return bad("spectra");
  if (cudaMalloc(&s->d_fmax, sizeof(float) * nk) != cudaSuccess) return bad("filter bound");
  cudaMemcpy(s->d_fmax, fmax.data(), sizeof(float) * nk, cudaMemcpyHostToDevice);
  if (cudaMalloc(&s->d_pscale, sizeof(float) * p.max_batch) != cudaSuccess) return bad("scales");
  const size_t pb = dtype_bytes(p.panel_dtype) * (size_t)p.nbins * p.nffti * p.max_batch;
  if (cudaMalloc(&s->d_panels, pb) != cudaSuccess) return bad("panels");
  if (cudaMalloc(&s->d_any, sizeof(int) * p.max_batch) != cudaSuccess) return bad("flags");
  s->form = p.form;
  if (p.form == QPSDM_FORM_BATCHED) {
    if (batched_alloc(s, p)) return bad("batched scratch");
  } else if (p.form != QPSDM_FORM_PLAIN) {
    if (err) *err = "unknown physics form";
    physics_destroy(s);
    return QPSDM_EINVAL;
  }
  *out = s;
  return QPSDM_OK;
}

void physics_destroy(PhysicsState *s) {
  if (!s) return;
  if (s->aux) cudaStreamSynchronize(s->aux);
  for (GroupSet &g : s->sets) {
    for (int i = 0; i < 2; ++i) {
      cudaFree(g.d_key[i]);
      cudaFree(g.d_val[i]);
    }
    cudaFree(g.d_ukey);
    cudaFree(g.d_count);
    cudaFree(g.d_off);
    cudaFree(g.d_nruns);
    cudaFree(g.d_srcflag);
    cudaFree(g.d_sid);
    cudaFree(g.d_srcpos);
    cudaFree(g.d_mem);
    cudaFree(g.d_grppos);
    cudaFree(g.d_memgrp);
    cudaFree(g.d_tile_ctr);
    cudaFree(g.d_defer);
    cudaFree(g.d_part);
    cudaFree(g.d_nmem);
    cudaFree(g.d_cub);
  }
  if (s->ev_fork) cudaEventDestroy(s->ev_fork);
  if (s->ev_join) cudaEventDestroy(s->ev_join);
  if (s->aux) cudaStreamDestroy(s->aux);
  cudaFree(s->d_filter);
  cudaFree(s->d_spec);
  cudaFree(s->d_fmax);
  cudaFree(s->d_pscale);
  cudaFree(s->d_panels);
  cudaFree(s->d_comp);
  for (auto &t : s->tabs) {
    cudaFree(t.dt);
    cudaFree(t.dq);
    cudaFree(t.ttt);
    cudaFree(t.qqq);
    cudaFree(t.tq);
  }
  cudaFree(s->d_any);
  cudaFree(s->d_tune);
  cudaFree(s->d_tab_tmp);
  delete s;
}

template <typename T>
static bool grow_dev(T **p, size_t *cap, size_t need) {
  if (*p && *cap >= need) return true;
  cudaFree(*p);
  *p = nullptr;
  *cap = 0;
  if (cudaMalloc((void **)p, sizeof(T) * (need ? need : 1)) != cudaSuccess) {
    cudaGetLastError();  // told by the result: the caller may have another way
    return false;
  }
  *cap = need;
  return true;
}

static int check_tables(const qpsdm_line_params &l, std::string *err) {
  if (!l.ttt_desc || !l.qqq_desc || !l.ttt || !l.qqq || l.nxg <= 0 || l.nzg <= 0 ||
      l.nxi1 <= 0 || l.nzi1 <= 0) {
    if (err) *err = "physics mode needs ttt and qqq tables";
    return QPSDM_EINVAL;
  }
  if (l.ttt_cdp1 > l.ttt_cdp2) {
    if (err) *err = "travel time table cdp range error";  // src/q-psdm.cu:1455-1461
    return QPSDM_EINVAL;
  }
  const size_t ncell = (size_t)l.nxg * l.nzg;
  // every descriptor's block must lie inside its data array
  for (int w = 0; w < 2; ++w) {
    const qpsdm_ttt_desc *d = w ? l.qqq_desc : l.ttt_desc;
    const int64_t len = w ? l.qqq_len : l.ttt_len;
    for (size_t c = 0; c < ncell; ++c) {
      const int64_t blk = (int64_t)d[c].nys * d[c].nxs * l.nxi1 * l.nzi1;
      if (d[c].idx < 0 || d[c].nys == 0 || d[c].nxs == 0 || d[c].dys == 0 ||
          d[c].dxs == 0 || d[c].idx + blk > len) {
        if (err) *err = "table descriptor outside its data (or empty surface grid)";
        return QPSDM_EINVAL;
      }
    }
  }
  return QPSDM_OK;
}

// Batched form: every surface node's [nxi1][nzi1] plane of a table cell
// (the reference layout, depth fastest) re-laid out as [nzi1][nxi1] (cdp
// fastest), so that image points of neighbouring cdps, which a warp of the
// batched kernel holds, read neighbouring table words.  Out of place:
// descriptors may share a block.  gridDim.y CTAs share the ncell cells.
__global__ void k_tab_xfast(const float *__restrict__ in, float *__restrict__ out,
                            const qpsdm_ttt_desc *__restrict__ desc, int ncell, int nxi1,
                            int nzi1) {
  const int plane = nxi1 * nzi1;
  for (int c = blockIdx.y; c < ncell; c += gridDim.y) {
    const qpsdm_ttt_desc d = desc[c];
    const int nplanes = (int)d.nys * d.nxs;
    for (int pl = blockIdx.x; pl < nplanes; pl += gridDim.x) {
      const int64_t base = d.idx + (int64_t)pl * plane;
      for (int e = threadIdx.x; e < plane; e += blockDim.x) {
        const int ixl = e / nzi1, izl = e - ixl * nzi1;
        out[base + izl * nxi1 + ixl] = in[base + e];
      }
    }
  }
}

// Two tables with identical descriptors as one array of (t, t*) of a node and
// (t, t*) of the node below it, cdp fastest (batched form) or in the tables' own
// order: a receiver's lookup at both depth nodes of a point is four 16-byte
// loads instead of eight 8-byte or sixteen 4-byte ones.  Below a cell's last
// node comes the first node of the cell under it (on the same surface grid;
// else, and below the deepest cell, the node itself, whose weight is zero).
// With one table null, the other's halves of the quads alone are written.
__global__ void k_tab_quads(const float *__restrict__ t, const float *__restrict__ q,
                            float4 *__restrict__ out, const qpsdm_ttt_desc *__restrict__ desc,
                            int ncell, int nzg, int nxi1, int nzi1, int xfast) {
  const int plane = nxi1 * nzi1;
  for (int c = blockIdx.y; c < ncell; c += gridDim.y) {
    const qpsdm_ttt_desc d = desc[c];
    const int nplanes = (int)d.nys * d.nxs;
    int64_t under = -1;
    if ((c + 1) % nzg != 0) {
      const qpsdm_ttt_desc e = desc[c + 1];
      if (e.nys == d.nys && e.nxs == d.nxs && e.dys == d.dys && e.dxs == d.dxs) under = e.idx;
    }
    for (int pl = blockIdx.x; pl < nplanes; pl += gridDim.x) {
      const int64_t base = d.idx + (int64_t)pl * plane, ub = under + (int64_t)pl * plane;
      for (int o = threadIdx.x; o < plane; o += blockDim.x) {
        const int izl = xfast ? o / nxi1 : o % nzi1;
        const int ixl = xfast ? o - izl * nxi1 : o / nzi1;
        const int64_t i = base + ixl * nzi1 + izl;
        const int64_t j = izl + 1 < nzi1 ? i + 1 : under >= 0 ? ub + ixl * nzi1 : i;
        float4 &w = out[base + o];
        if (t && q)
          w = make_float4(t[i], q[i], t[j], q[j]);
        else if (t)
          w.x = t[i], w.z = t[j];
        else
          w.y = q[i], w.w = q[j];
      }
    }
  }
}

// Whether one quad per table entry serves every cell of a line that reads the
// entry: blocks that overlap have their planes at the same places, and the node
// under their last one equally far on (cells that share a v(z) table column by
// column do; blocks shared by cells of different depths do not).
static bool quads_fit(const qpsdm_line_params &l) {
  struct Block {
    int64_t lo, hi, under;
  };
  const int64_t plane = (int64_t)l.nxi1 * l.nzi1;
  std::vector<Block> b((size_t)l.nxg * l.nzg);
  for (size_t c = 0; c < b.size(); ++c) {
    const qpsdm_ttt_desc &d = l.ttt_desc[c];
    b[c] = {d.idx, d.idx + (int64_t)d.nys * d.nxs * plane, INT64_MIN};
    if ((c + 1) % l.nzg != 0) {
      const qpsdm_ttt_desc &e = l.ttt_desc[c + 1];
      if (e.nys == d.nys && e.nxs == d.nxs && e.dys == d.dys && e.dxs == d.dxs)
        b[c].under = e.idx - d.idx;
    }
  }
  std::sort(b.begin(), b.end(), [](const Block &x, const Block &y) { return x.lo < y.lo; });
  Block far = b[0];  // of the blocks so far, the one that ends last
  for (const Block &x : b) {
    if (x.lo < far.hi && ((x.lo - far.lo) % plane != 0 || x.under != far.under)) return false;
    if (x.hi > far.hi) far = x;
  }
  return true;
}

// Tables of a brick's lines; (t, t*) quads where `pair` and the tables allow it.
static int upload_lines(PhysicsState *s, const qpsdm_line_params *lines, int nlines, bool pair,
                        cudaStream_t st) {
  int dev = 0;
  cudaGetDevice(&dev);
  // data already in this device's memory is read in place
  auto on_device = [dev](const float *p) {
    cudaPointerAttributes at;
    const bool yes = cudaPointerGetAttributes(&at, p) == cudaSuccess &&
                     at.type == cudaMemoryTypeDevice && at.device == dev;
    cudaGetLastError();  // a pageable pointer may leave an error behind
    return yes;
  };
  const bool batched = s->form == QPSDM_FORM_BATCHED;
  for (int il = 0; il < nlines; ++il) {
    const qpsdm_line_params &l = lines[il];
    PhysicsState::LineTab &t = s->tabs[il];
    const size_t ncell = (size_t)l.nxg * l.nzg;
    t.one_grid = true;
    for (size_t c = 0; c < ncell && t.one_grid; ++c)
      t.one_grid = l.ttt_desc[c].nxs == l.ttt_desc[0].nxs &&
                   l.ttt_desc[c].nys == l.ttt_desc[0].nys &&
                   l.ttt_desc[c].dxs == l.ttt_desc[0].dxs &&
                   l.ttt_desc[c].dys == l.ttt_desc[0].dys &&
                   (int64_t)l.ttt_desc[c].nxs * l.ttt_desc[c].nys * l.nxi1 * l.nzi1 < (1ll << 30);
    // identical descriptors (the reference writes both tables alike): t and t*
    // of a node are read together
    t.paired = pair && l.ttt_len == l.qqq_len &&
               std::memcmp(l.ttt_desc, l.qqq_desc, sizeof(qpsdm_ttt_desc) * ncell) == 0 &&
               quads_fit(l);
    // paired tables on one surface grid need no table of their own
    const bool single = !(t.paired && t.one_grid);
    if (!grow_dev(&t.dt, &t.dt_cap, ncell) || !grow_dev(&t.dq, &t.dq_cap, ncell) ||
        (single && (!grow_dev(&t.ttt, &t.ttt_cap, (size_t)l.ttt_len) ||
                    !grow_dev(&t.qqq, &t.qqq_cap, (size_t)l.qqq_len))) ||
        (t.paired && !grow_dev(&t.tq, &t.tq_cap, (size_t)l.ttt_len)))
      return QPSDM_ENOMEM;
    cudaMemcpyAsync(t.dt, l.ttt_desc, sizeof(qpsdm_ttt_desc) * ncell, cudaMemcpyHostToDevice, st);
    cudaMemcpyAsync(t.dq, l.qqq_desc, sizeof(qpsdm_ttt_desc) * ncell, cudaMemcpyHostToDevice, st);
    const int nc = (int)ncell;  // cells past a grid's 65,535 rows come in turn
    const dim3 g(256, (unsigned)std::min(nc, 65535));
    // a table in host memory passes through the staging copy, one after the other
    const bool both = on_device(l.ttt) && on_device(l.qqq);
    for (int w = 0; w < 2; ++w) {
      const float *src = w ? l.qqq : l.ttt;
      const size_t len = (size_t)(w ? l.qqq_len : l.ttt_len);
      float *own = w ? t.qqq : t.ttt;
      const qpsdm_ttt_desc *d = w ? t.dq : t.dt;
      if (single && !batched)
        cudaMemcpyAsync(own, src, sizeof(float) * len, cudaMemcpyDefault, st);
      if (!t.paired && !batched) continue;
      if (!both && !on_device(src)) {
        if (!grow_dev(&s->d_tab_tmp, &s->tab_tmp_cap, len)) return QPSDM_ENOMEM;
        cudaMemcpyAsync(s->d_tab_tmp, src, sizeof(float) * len, cudaMemcpyDefault, st);
        src = s->d_tab_tmp;
      }
      if (t.paired && (!both || w == 0))
        k_tab_quads<<<g, 256, 0, st>>>(w ? nullptr : src, both ? l.qqq : w ? src : nullptr, t.tq,
                                       d, nc, l.nzg, l.nxi1, l.nzi1, batched);
      if (single && batched) k_tab_xfast<<<g, 256, 0, st>>>(src, own, d, nc, l.nxi1, l.nzi1);
    }
  }
  return QPSDM_OK;
}

template <typename T>
static void free_dev(T **p, size_t *cap) {
  cudaFree(*p);
  *p = nullptr;
  *cap = 0;
}

// Table data may be host memory or memory of the engine's device; descriptors
// are host memory.  Quads take 16 bytes an entry (24 beside the float tables,
// with several surface grids); where they do not fit the GPU, every line gets
// float tables alone, 8 bytes.
int physics_set_lines(PhysicsState *s, const qpsdm_static_params &p,
                      const qpsdm_line_params *lines, int nlines, cudaStream_t st,
                      std::string *err) {
  (void)p;
  for (int il = 0; il < nlines; ++il) {
    int rc = check_tables(lines[il], err);
    if (rc) return rc;
  }
  if ((int)s->tabs.size() < nlines) s->tabs.resize(nlines);
  int rc = upload_lines(s, lines, nlines, true, st);
  if (rc == QPSDM_ENOMEM) {
    cudaStreamSynchronize(st);
    for (PhysicsState::LineTab &t : s->tabs) {
      free_dev(&t.ttt, &t.ttt_cap);
      free_dev(&t.qqq, &t.qqq_cap);
      free_dev(&t.tq, &t.tq_cap);
    }
    free_dev(&s->d_tab_tmp, &s->tab_tmp_cap);
    s->ntabs = 0;
    rc = upload_lines(s, lines, nlines, false, st);
  }
  if (rc) {
    cudaStreamSynchronize(st);
    if (err) *err = "table allocation failed";
    return rc;
  }
  if (cudaGetLastError() != cudaSuccess || cudaStreamSynchronize(st) != cudaSuccess) {
    if (err) *err = "table upload failed";
    return QPSDM_ECUDA;
  }
  // the plain form's staging copy: a small one is kept for the next lines
  if (s->form == QPSDM_FORM_PLAIN && s->tab_tmp_cap > kTabTmpKeep)
    free_dev(&s->d_tab_tmp, &s->tab_tmp_cap);
  s->ntabs = nlines;
  return QPSDM_OK;
}

int physics_begin_offset(PhysicsState *s, const qpsdm_static_params &p,
                         const qpsdm_offset_params &o, int nlines, cudaStream_t st,
                         std::string *err) {
  if (s->form == QPSDM_FORM_BATCHED && s->variant < 0 &&
      !grow_dev(&s->d_tune, &s->tune_cap, (size_t)(o.ixend - o.ixstart) * p.nzi)) {
    if (err) *err = "autotuner scratch allocation failed";
    return QPSDM_ENOMEM;
  }
  if (s->form == QPSDM_FORM_BATCHED) {
    const size_t nxb = (size_t)(o.ixend - o.ixstart);
    const size_t npt = nxb * p.nzi, ntile = npt / 32 + nxb + p.nzi + 1;  // tiles: 32 points or more
    for (GroupSet &g : s->sets) {
      if (!grow_dev(&g.d_defer, &g.defer_cap, ntile) ||
          !grow_dev(&g.d_tile_ctr, &g.ctr_cap, 2 + ntile)) {
        if (err) *err = "tile queue allocation failed";
        return QPSDM_ENOMEM;
      }
      g.d_ndefer = g.d_tile_ctr + 1;
    }
  }
  if (p.kahan) {
    const size_t n = (size_t)(o.ixend - o.ixstart) * p.nzi * nlines;
    if (!grow_dev(&s->d_comp, &s->comp_cap, n)) {
      if (err) *err = "compensation buffer allocation failed";
      return QPSDM_ENOMEM;
    }
    cudaMemsetAsync(s->d_comp, 0, sizeof(float) * n, st);
  }
  if (s->form == QPSDM_FORM_BATCHED) {
    // without room for the parts' sums no tile is split (member_split)
    const size_t npt = (size_t)(o.ixend - o.ixstart) * p.nzi;
    for (GroupSet &g : s->sets)
      grow_dev(&g.d_part, &g.part_cap, std::min(kMaxSplit * npt, kSplitSums) * s->part_words);
    select_set(s, s->cur_set);
  }
  return QPSDM_OK;
}

// ---------------------------------------------------------------------------
// panels
// ---------------------------------------------------------------------------
__device__ __forceinline__ float phys_tapered(float v, int j, int n, const float *tap) {
  const int head = j, tail = n - 1 - j;
  if (head < 200 && tail < 200) {
    if (head <= tail) return __fmul_rn(__fmul_rn(v, tap[head]), tap[tail]);
    return __fmul_rn(__fmul_rn(v, tap[tail]), tap[head]);
  }
  if (head < 200) return __fmul_rn(v, tap[head]);
  if (tail < 200) return __fmul_rn(v, tap[tail]);
  return v;
}

// Gained and tapered sample j of a trace (zero beyond its end).
__device__ __forceinline__ float phys_sample(const uint8_t *r, int j, int be, int ntl, float dt,
                                             const float *tap) {
  if (j >= ntl) return 0.0f;
  float v = su_sample(r, j, be);
  const float t = __fmul_rn((float)j, dt);
  v = ((double)t < 0.1) ? __double2float_rn(__dmul_rn((double)v, 0.1 * 0.1))
                        : __fmul_rn(v, __fmul_rn(t, t));
  return phys_tapered(v, j, ntl, tap);
}

// Forward spectra of the accepted traces, two neighbouring traces per CTA
// (fft.cuh).  For FP16 panels also the trace's sample multiplier: every panel
// sample of the trace is bounded by B = 2 sum_k |X_k| max_b |F_b,k| (triangle
// inequality over the c2r sum), and the panels store x / 2^e with e chosen so
// that B / 2^e lies in [2^13, 2^14): no overflow of FP16 (max 65504) and no
// loss to its subnormal range; the image kernels multiply the samples by 2^e
// again (exact).
template <bool PAD>
__global__ void __launch_bounds__(kFftMaxThreads, 2)
    k_phys_fwd(const uint8_t *__restrict__ rec, int rec_bytes, int be,
               const int *__restrict__ status, int sstride, int ntr, int ntl, float dt,
               const float *__restrict__ tap, const __grid_constant__ FftPlan p,
               float2 *__restrict__ spec, const float *__restrict__ fmax,
               float *__restrict__ pscale) {
  extern __shared__ float4 pbuf[];
  __shared__ float s_part[2][kFftMaxThreads / 32];
  const int ia = 2 * blockIdx.x, ib = min(ia + 1, ntr - 1);
  const bool oka = status[(size_t)ia * sstride] == kAccepted;
  const bool okb = ib != ia && status[(size_t)ib * sstride] == kAccepted;
  if (!oka && !okb) return;  // uniform in the CTA
  const uint8_t *ra = rec + (size_t)ia * rec_bytes, *rb = rec + (size_t)ib * rec_bytes;
  for (int j = threadIdx.x; j < p.m; j += blockDim.x) {
    float4 v;
    v.x = phys_sample(ra, 2 * j, be, ntl, dt, tap);
    v.y = phys_sample(rb, 2 * j, be, ntl, dt, tap);
    v.z = phys_sample(ra, 2 * j + 1, be, ntl, dt, tap);
    v.w = phys_sample(rb, 2 * j + 1, be, ntl, dt, tap);
    pbuf[stock_slot<PAD>(j)] = v;
  }
  __syncthreads();
  const float4 *Z = stock_passes<false, PAD>(pbuf, pbuf, p, 0, p.nstock);
  float2 *oa = spec + (size_t)ia * (p.m + 1), *ob = spec + (size_t)ib * (p.m + 1);
  float ba = 0.0f, bb = 0.0f;
  auto put = [&](int k, C2 v) {
    const float2 re = f2_unpack(v.re), im = f2_unpack(v.im);
    if (oka) oa[k] = make_float2(re.x, im.x);
    if (okb) ob[k] = make_float2(re.y, im.y);
    if (pscale) {
      const float f = fmax[k];
      ba = fmaf(sqrtf(re.x * re.x + im.x * im.x), f, ba);
      bb = fmaf(sqrtf(re.y * re.y + im.y * im.y), f, bb);
    }
  };
  for (int k = threadIdx.x; 2 * k <= p.m; k += blockDim.x) {
    const int k2 = p.m - k;
    C2 u, v;
    pfa_rfft_bins(pfa_ld(Z, stock_slot<PAD>(k)), pfa_ld(Z, stock_slot<PAD>(k ? k2 : 0)),
                  __ldg(p.tw_n + k), u, v);
    put(k, u);
    if (k2 != k) put(k2, v);
  }
  if (!pscale) return;
  for (int off = 16; off > 0; off >>= 1) {
    ba += __shfl_xor_sync(0xffffffffu, ba, off);
    bb += __shfl_xor_sync(0xffffffffu, bb, off);
  }
  if ((threadIdx.x & 31) == 0) {
    s_part[0][threadIdx.x >> 5] = ba;
    s_part[1][threadIdx.x >> 5] = bb;
  }
  __syncthreads();
  if (threadIdx.x < 2 && (threadIdx.x ? okb : oka)) {
    float b = 0.0f;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) b += s_part[threadIdx.x][w];
    b *= 2.0f;
    int e = 0;
    if (b > 0.0f && isfinite(b)) {
      frexpf(b, &e);  // b = m 2^e, m in [0.5, 1)
      e = min(max(e - 14, -126), 127);
    }
    pscale[threadIdx.x ? ib : ia] = ldexpf(1.0f, e);
  }
}

// Two neighbouring samples of a panel row (rows have even lengths).
__device__ __forceinline__ void store_two(float *d, float a, float b) {
  *reinterpret_cast<float2 *>(d) = make_float2(a, b);
}
__device__ __forceinline__ void store_two(__half *d, float a, float b) {
  *reinterpret_cast<__half2 *>(d) = __floats2half2_rn(a, b);
}
__device__ __forceinline__ void store_two(__nv_bfloat16 *d, float a, float b) {
  *reinterpret_cast<__nv_bfloat162 *>(d) = __floats2bfloat162_rn(a, b);
}

// t*-binned panels: for every accepted trace and bin b, the filtered,
// zero-padded spectrum X F_b -> c2r of length nffti.  Two bins share every
// instruction of the inverse transform (fft.cuh); kmax is the first frequency
// bin past the band, where every F_b is zero.  A CTA takes (trace, group of
// bin pairs) items, keeps the band of the trace's spectrum in shared memory
// and runs its pairs back to back.  The first group of passes computes its
// own inputs, a butterfly and its mirror image together (one filtered pair
// Y[k], Y[m-k] gives both Z[k] and Z[m-k] of the c2r split), and the last
// radix stores its outputs to the panel (neighbouring butterflies have
// neighbouring outputs): a point crosses shared memory six times for
// m = 3003 = 3 x 7 x 11 x 13, not ten.  With one bin per instruction, the roots
// and twiddles in shared memory: 8.97 ms with the forward transforms for 24,902
// traces of m = 2520, 6.37 ms for 30,000 of m = 3003, 4.80 ms for 18,432 of
// m = 2002; now 5.2, 4.0 and 3.8 ms.  Two CTAs an SM (two 48 KB buffers each,
// 96 registers a thread) leave it waiting for twiddles and barriers: issue
// active 44 %.  The passes round like those of a
// scalar transform in the same order, so a panel's half-precision values do
// not depend on how the transform is packed or grouped.
template <bool PAD, typename T>
__global__ void __launch_bounds__(kFftMaxThreads, 2)
    k_phys_panels(const int *__restrict__ status, int sstride, int ntr,
                  const float2 *__restrict__ spec, int nk, int kmax,
                  const float4 *__restrict__ filt, const __grid_constant__ FftPlan p, int nbins,
                  int ngroups, T *__restrict__ panels, const float *__restrict__ pscale) {
  extern __shared__ float4 pbuf[];
  const int m = p.m;
  float2 *Xs = reinterpret_cast<float2 *>(pbuf + 2 * p.swords);
  const int npairs = (nbins + 1) / 2, per = (npairs + ngroups - 1) / ngroups;
  // fused first group and last radix: up to 8 points a butterfly, and two
  // groups at least
  const int code0 = p.nstock > 1 ? p.stock[0] : 0, code1 = p.nstock > 1 ? p.stock[p.nstock - 1] : 0;
  const bool fuse_in = p.nstock > 1 && (code0 & 15) * (code0 >> 4) <= 8;
  const bool fuse_out = p.nstock > 1 && code1 >> 4 == 1;
  for (int item = blockIdx.x; item < ntr * ngroups; item += gridDim.x) {
    const int itr = item / ngroups, bp0 = (item - itr * ngroups) * per;
    if (status[(size_t)itr * sstride] != kAccepted) continue;  // uniform in the CTA
    const float2 *X = spec + (size_t)itr * nk;
    for (int k = threadIdx.x; k < kmax; k += blockDim.x) Xs[k] = X[k];
    __syncthreads();
    // 2 / 2^e for FP16 (exact), 2 otherwise
    const float mul = std::is_same<T, __half>::value ? 2.0f / pscale[itr] : 2.0f;
    for (int bp = bp0; bp < min(bp0 + per, npairs); ++bp) {
      const float4 *F = filt + (size_t)bp * kmax;
      // filtered bin k of both, zero past the band
      auto bin = [&](int k) {
        C2 y{0ull, 0ull};
        if (k < kmax) {
          const float2 x = Xs[k];
          const float4 f = __ldg(F + k);
          const f2 fr = f2_pack(f.x, f.y), fi = f2_pack(f.z, f.w);
          y.re = f2_fma(f2_dup(x.x), fr, f2_mul(f2_dup(-x.y), fi));
          y.im = f2_fma(f2_dup(x.x), fi, f2_mul(f2_dup(x.y), fr));
        }
        return y;
      };
      float4 *in = pbuf;
      if (fuse_in) {
        stock_by_code(code0, [&](auto cA, auto cB) {
          constexpr int PA = decltype(cA)::value, PB = decltype(cB)::value, Q = PA * PB;
          if constexpr (Q <= 8) {
            const int M = m / Q;
            auto put = [&](int n, C2 o) { pfa_st(pbuf, stock_slot<PAD>(n), o); };
            for (int J = threadIdx.x; 2 * J <= M; J += blockDim.x) {
              C2 u[Q], v[Q];
#pragma unroll
              for (int i = 0; i < Q; ++i) {
                const int k = J + i * M;
                pfa_irfft_pre(bin(k), bin(m - k), __ldg(p.tw_n + k), u[i], v[Q - 1 - i]);
              }
              stock_group<PA, PB, true>(u, J, m, 1, 0u, p.tw_m, put);
              // butterfly 0 mirrors itself, as does the middle one
              if (J > 0 && 2 * J < M) stock_group<PA, PB, true>(v, M - J, m, 1, 0u, p.tw_m, put);
            }
          }
        });
      } else {
        for (int k = threadIdx.x; 2 * k <= m; k += blockDim.x) {
          const int k2 = m - k;
          C2 u, v;
          pfa_irfft_pre(bin(k), bin(k2), __ldg(p.tw_n + k), u, v);
          pfa_st(pbuf, stock_slot<PAD>(k), u);
          if (k > 0 && k < k2) pfa_st(pbuf, stock_slot<PAD>(k2), v);
        }
      }
      __syncthreads();
      in = stock_passes<true, PAD>(pbuf, in, p, fuse_in ? 1 : 0, p.nstock - (fuse_out ? 1 : 0));
      T *out = panels + ((size_t)itr * nbins + 2 * bp) * p.n;
      const bool two = 2 * bp + 1 < nbins;
      auto store = [&](int n, C2 z) {
        const float2 re = f2_unpack(z.re), im = f2_unpack(z.im);
        store_two(out + 2 * n, mul * re.x, mul * im.x);
        if (two) store_two(out + p.n + 2 * n, mul * re.y, mul * im.y);
      };
      if (fuse_out) {
        stock_by_code(code1, [&](auto cA, auto cB) {
          constexpr int PA = decltype(cA)::value;
          if constexpr (decltype(cB)::value == 1)
            stock_pass<PA, 1, true, PAD>(in, m, m / PA, p.tw_m, store);
        });
      } else {
        for (int j = threadIdx.x; j < m; j += blockDim.x) store(j, pfa_ld(in, stock_slot<PAD>(j)));
      }
      __syncthreads();  // the next pair writes pbuf (and the next item Xs)
    }
  }
}

// ---------------------------------------------------------------------------
// plain imaging
// ---------------------------------------------------------------------------
struct PhysImageArgs {
  int nzi, nxb, ixstart, nt, nbins;
  float dt1, dxi, dzi, taperzone, dtstar, dzii;
  int tcdp1, tcdp2;  // relative to fci
  int nxg, nzg, nxi1, nzi1;
  size_t nxz;
  int xfast;  // tables stored [izl][ixl] inside each surface node's plane (batched form)
};

template <typename T>
__device__ __forceinline__ float ld_sample(const T *p);
template <>
__device__ __forceinline__ float ld_sample<float>(const float *p) { return __ldg(p); }
template <>
__device__ __forceinline__ float ld_sample<__nv_bfloat16>(const __nv_bfloat16 *p) {
  return __bfloat162float(*p);
}
template <>
__device__ __forceinline__ float ld_sample<__half>(const __half *p) { return __half2float(*p); }

// a + w (b - a) as one fused multiply-add (the form every table and sample
// interpolation of the image kernels takes; the FP32 oracle repeats it).
__device__ __forceinline__ float lerp(float a, float b, float w) {
  return __fmaf_rn(w, __fsub_rn(b, a), a);
}

// a + w (b - a) of a (t, t*) pair, both halves with one instruction each.
__device__ __forceinline__ f2 f2_lerp(f2 a, f2 b, f2 w) { return f2_fma(w, f2_sub(b, a), a); }
// Bilinear (t, t*) at a point's two depth nodes (v[0] the upper) from the 2 x 2
// surface nodes n (bilin's arithmetic, halves packed).
__device__ __forceinline__ void bilin_tq(const ulonglong2 (&n)[4], f2 wx, f2 wy, f2 (&v)[2]) {
  v[0] = f2_lerp(f2_lerp(n[0].x, n[1].x, wx), f2_lerp(n[2].x, n[3].x, wx), wy);
  v[1] = f2_lerp(f2_lerp(n[0].y, n[1].y, wx), f2_lerp(n[2].y, n[3].y, wx), wy);
}
__device__ __forceinline__ void load_nodes(const float4 *__restrict__ p, int sx, int sy,
                                           ulonglong2 (&n)[4]) {
  const ulonglong2 *q = reinterpret_cast<const ulonglong2 *>(p);
  n[0] = __ldg(q), n[1] = __ldg(q + sx);
  n[2] = __ldg(q + sy), n[3] = __ldg(q + (sy + sx));
}

// Bilinear value of a 2 x 2 node block starting at tab + base.
__device__ __forceinline__ float bilin(const float *__restrict__ tab, int64_t base, int64_t sx,
                                       int64_t sy, float wx, float wy) {
  const float v00 = __ldg(tab + base), v01 = __ldg(tab + base + sx);
  const float v10 = __ldg(tab + base + sy), v11 = __ldg(tab + base + sy + sx);
  return lerp(lerp(v00, v01, wx), lerp(v10, v11, wx), wy);
}

// Table value at one depth node of a cell for surface point (px, py).
// Returns false outside the cell's surface grid.
__device__ __forceinline__ bool table_node(const qpsdm_ttt_desc &d, const float *__restrict__ tab,
                                           float px, float py, float xc, int poff,
                                           int nxi1, int nzi1, float &v) {
  const int nxs = d.nxs, nys = d.nys;
  float fx, fy;
  if (!grid_pos(px, py, xc, __fdiv_rn(1.0f, (float)d.dxs), __fdiv_rn(1.0f, (float)d.dys),
                0.5f * (nxs - 1), 0.5f * (nys - 1), nxs, nys, fx, fy))
    return false;
  int ix = min((int)fx, max(nxs - 2, 0));
  int iy = min((int)fy, max(nys - 2, 0));
  const float wx = nxs > 1 ? __fsub_rn(fx, (float)ix) : 0.0f;
  const float wy = nys > 1 ? __fsub_rn(fy, (float)iy) : 0.0f;
  const int64_t sx = nxs > 1 ? (int64_t)nxi1 * nzi1 : 0;
  const int64_t sy = nys > 1 ? (int64_t)nxs * nxi1 * nzi1 : 0;
  const int64_t base = d.idx + (int64_t)(iy * nxs + ix) * nxi1 * nzi1 + poff;
  v = bilin(tab, base, sx, sy, wx, wy);
  return true;
}

struct PointCells {
  bool ok;
  bool same;  // all four descriptors share one surface grid
  int offA, offB;       // offsets of the point's two depth nodes inside a surface plane
  int cA, cB;          // cells of the two depth nodes
  int nxs, nys;        // shared surface grid (fast path)
  float c2, xc;
  float rdx, rdy, hx, hy;  // 1/dxs, 1/dys, (nxs-1)/2, (nys-1)/2 of the shared grid
  int64_t tA, tB, qA, qB;  // data offsets (idx) of the four blocks
};

__device__ __forceinline__ bool same_grid(const qpsdm_ttt_desc &a, const qpsdm_ttt_desc &b) {
  return a.nxs == b.nxs && a.nys == b.nys && a.dxs == b.dxs && a.dys == b.dys;
}

// Cell, depth node and descriptors of image point (ixi, z), src/q-psdm.cu:2343-2349.
__device__ __forceinline__ void setup_cells(PointCells &pc, int ixi, float z,
                                            const PhysImageArgs &a,
                                            const qpsdm_ttt_desc *__restrict__ dt,
                                            const qpsdm_ttt_desc *__restrict__ dq) {
  pc.ok = false;
  pc.same = false;
  if (ixi < a.tcdp1 || ixi > a.tcdp2) return;
  const int lx = ixi - a.tcdp1;
  const int ixg = lx / a.nxi1;
  const int ixl = lx - ixg * a.nxi1;
  const float fz = __fdiv_rn(z, a.dzii);
  const int izn = (int)fz;
  pc.c2 = __fsub_rn(fz, (float)izn);
  int izgA = izn / a.nzi1, izgB = (izn + 1) / a.nzi1;
  int izlA = izn - izgA * a.nzi1;
  int izlB = izn + 1 - izgB * a.nzi1;
  if (izgB >= a.nzg) {  // deepest node: no lower neighbour
    izgB = izgA;
    izlB = izlA;
    pc.c2 = 0.0f;
  }
  if (ixg >= a.nxg || izgA >= a.nzg) return;
  pc.ok = true;
  // [ixl][izl] planes (the reference layout) or [izl][ixl] (batched form)
  pc.offA = a.xfast ? izlA * a.nxi1 + ixl : ixl * a.nzi1 + izlA;
  pc.offB = a.xfast ? izlB * a.nxi1 + ixl : ixl * a.nzi1 + izlB;
  pc.cA = ixg * a.nzg + izgA;
  pc.cB = ixg * a.nzg + izgB;
  const qpsdm_ttt_desc tA = dt[pc.cA], tB = dt[pc.cB], qA = dq[pc.cA], qB = dq[pc.cB];
  pc.tA = tA.idx;
  pc.tB = tB.idx;
  pc.qA = qA.idx;
  pc.qB = qB.idx;
  pc.xc = __fmul_rn(__fadd_rn((float)(a.tcdp1 + ixg * a.nxi1), 0.5f * (a.nxi1 - 1)), a.dxi);
  pc.same = same_grid(tA, tB) && same_grid(tA, qA) && same_grid(tA, qB);
  pc.nxs = tA.nxs;
  pc.nys = tA.nys;
  pc.rdx = __fdiv_rn(1.0f, (float)tA.dxs);
  pc.rdy = __fdiv_rn(1.0f, (float)tA.dys);
  pc.hx = 0.5f * (tA.nxs - 1);
  pc.hy = 0.5f * (tA.nys - 1);
}


__device__ __forceinline__ bool lookup_tq(const PointCells &pc,
                                          const qpsdm_ttt_desc *__restrict__ dt,
                                          const float *__restrict__ ttt,
                                          const qpsdm_ttt_desc *__restrict__ dq,
                                          const float *__restrict__ qqq, int nxi1, int nzi1,
                                          float px, float py, float &t, float &q) {
  if (pc.same) {  // one set of surface weights for t and t*, both depth nodes
    const int nxs = pc.nxs, nys = pc.nys;
    float fx, fy;
    if (!grid_pos(px, py, pc.xc, pc.rdx, pc.rdy, pc.hx, pc.hy, nxs, nys, fx, fy)) return false;
    const int ix = min((int)fx, max(nxs - 2, 0));
    const int iy = min((int)fy, max(nys - 2, 0));
    const float wx = nxs > 1 ? __fsub_rn(fx, (float)ix) : 0.0f;
    const float wy = nys > 1 ? __fsub_rn(fy, (float)iy) : 0.0f;
    const int64_t plane = (int64_t)nxi1 * nzi1;
    const int64_t sx = nxs > 1 ? plane : 0, sy = nys > 1 ? (int64_t)nxs * plane : 0;
    const int64_t off = (int64_t)(iy * nxs + ix) * plane;
    const float ta = bilin(ttt, pc.tA + off + pc.offA, sx, sy, wx, wy);
    const float tb = bilin(ttt, pc.tB + off + pc.offB, sx, sy, wx, wy);
    const float qa = bilin(qqq, pc.qA + off + pc.offA, sx, sy, wx, wy);
    const float qb = bilin(qqq, pc.qB + off + pc.offB, sx, sy, wx, wy);
    t = lerp(ta, tb, pc.c2);
    q = lerp(qa, qb, pc.c2);
    return true;
  }
  // cells with different surface grids: one lookup per descriptor
  float ta, tb, qa, qb;
  if (!table_node(dt[pc.cA], ttt, px, py, pc.xc, pc.offA, nxi1, nzi1, ta)) return false;
  if (!table_node(dt[pc.cB], ttt, px, py, pc.xc, pc.offB, nxi1, nzi1, tb)) return false;
  if (!table_node(dq[pc.cA], qqq, px, py, pc.xc, pc.offA, nxi1, nzi1, qa)) return false;
  if (!table_node(dq[pc.cB], qqq, px, py, pc.xc, pc.offB, nxi1, nzi1, qb)) return false;
  t = lerp(ta, tb, pc.c2);
  q = lerp(qa, qb, pc.c2);
  return true;
}

// lookup_tq for a line whose t and t* tables have identical descriptors,
// read as (t, t*) pairs (tq): same values, same arithmetic, half the loads.
__device__ __forceinline__ float2 bilin2(const float4 *__restrict__ tab, int64_t base, int64_t sx,
                                         int64_t sy, float wx, float wy) {
  auto ld = [&](int64_t i) { return __ldg(reinterpret_cast<const float2 *>(tab + i)); };
  const float2 v00 = ld(base), v01 = ld(base + sx);
  const float2 v10 = ld(base + sy), v11 = ld(base + sy + sx);
  return make_float2(lerp(lerp(v00.x, v01.x, wx), lerp(v10.x, v11.x, wx), wy),
                     lerp(lerp(v00.y, v01.y, wx), lerp(v10.y, v11.y, wx), wy));
}
__device__ __forceinline__ bool lookup_tq(const PointCells &pc,
                                          const qpsdm_ttt_desc *__restrict__ dt,
                                          const float *__restrict__ ttt,
                                          const qpsdm_ttt_desc *__restrict__ dq,
                                          const float *__restrict__ qqq,
                                          const float4 *__restrict__ tq, int nxi1, int nzi1,
                                          float px, float py, float &t, float &q) {
  if (!tq || !pc.same) return lookup_tq(pc, dt, ttt, dq, qqq, nxi1, nzi1, px, py, t, q);
  const int nxs = pc.nxs, nys = pc.nys;
  float fx, fy;
  if (!grid_pos(px, py, pc.xc, pc.rdx, pc.rdy, pc.hx, pc.hy, nxs, nys, fx, fy)) return false;
  const int ix = min((int)fx, max(nxs - 2, 0));
  const int iy = min((int)fy, max(nys - 2, 0));
  const float wx = nxs > 1 ? __fsub_rn(fx, (float)ix) : 0.0f;
  const float wy = nys > 1 ? __fsub_rn(fy, (float)iy) : 0.0f;
  const int64_t plane = (int64_t)nxi1 * nzi1;
  const int64_t sx = nxs > 1 ? plane : 0, sy = nys > 1 ? (int64_t)nxs * plane : 0;
  const int64_t off = (int64_t)(iy * nxs + ix) * plane;
  const float2 a = bilin2(tq, pc.tA + off + pc.offA, sx, sy, wx, wy);
  const float2 b = bilin2(tq, pc.tB + off + pc.offB, sx, sy, wx, wy);
  t = lerp(a.x, b.x, pc.c2);
  q = lerp(a.y, b.y, pc.c2);
  return true;
}

// Per-launch counters cnt[0..2] += the block's per-thread counts: point-traces
// (pairs in the aperture with table values at both ends), of which decided
// for a whole tile (members dropped before any point saw them), and imaged
// (past the dip test and the time window).  One atomic per counter and block.
__device__ __forceinline__ void add_counts(unsigned long long *cnt, unsigned long long *s,
                                           unsigned c0, unsigned c1, unsigned c2) {
  const int tid = threadIdx.x + threadIdx.y * blockDim.x;
  const int nthr = blockDim.x * blockDim.y;
  if (tid < 3) s[tid] = 0;
  __syncthreads();
  for (int off = 16; off > 0; off >>= 1) {
    c0 += __shfl_down_sync(0xffffffffu, c0, off);
    c1 += __shfl_down_sync(0xffffffffu, c1, off);
    c2 += __shfl_down_sync(0xffffffffu, c2, off);
  }
  if ((tid & 31) == 0) {
    if (c0) atomicAdd(&s[0], (unsigned long long)c0);
    if (c1) atomicAdd(&s[1], (unsigned long long)c1);
    if (c2) atomicAdd(&s[2], (unsigned long long)c2);
  }
  __syncthreads();
  if (tid < 3 && s[tid]) atomicAdd(cnt + tid, s[tid]);
  (void)nthr;
}

// Plain imaging: each point sums its traces in submission order (ordered.cuh).
// In a tile whose points read the same table cells of paired tables coverage
// is decided per trace, and the surface weights of its receiver are computed
// once (uni); in any other tile the points look up and count for themselves.
// The table lookups come after the dip test, which fails for most pairs.
//
// Measured: 9,216 traces into a 512 x 400 line (8.3e8 point-traces, 2.2e8
// imaged) 12.7 ms with one thread running over every trace, the lookups before
// the test and every tangent divided out; 5.6 ms now, 128 registers, two blocks
// an SM, issue active 42 % (fixed-latency chains of the IEEE divisions and
// square roots first).  Three blocks at 85 registers were slower.
template <int SPLIT, typename T>
__global__ void __launch_bounds__(256)
    k_image_plain(float *__restrict__ img, float *__restrict__ comp, PhysImageArgs a,
                  const float *__restrict__ dips, const int *__restrict__ ints,
                  const float *__restrict__ geom, int ntr,
                  const qpsdm_ttt_desc *__restrict__ dt, const float *__restrict__ ttt,
                  const qpsdm_ttt_desc *__restrict__ dq, const float *__restrict__ qqq,
                  const float4 *__restrict__ tq, const T *__restrict__ panels,
                  const float *__restrict__ pscale, unsigned long long *npt) {
  constexpr int TX = 8 / SPLIT;
  __shared__ OrderedSmem<SPLIT> sm;
  __shared__ float s_red[13][8];
  __shared__ TileBox s_box;
  __shared__ TileGrid s_tg;
  __shared__ int s_tgw, s_col[TX];
  __shared__ unsigned long long s_cnt[3];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int iz0 = blockIdx.x * 32, ixb0 = blockIdx.y * TX, lx = warp / SPLIT;
  const int izi = iz0 + lane, ixb = ixb0 + lx;
  const bool live = izi < a.nzi && ixb < a.nxb, sums = SPLIT == 1 || warp % SPLIT == 0;
  const int ixi = ixb + a.ixstart;
  if (tid == 0) s_tgw = -1;

  // per-point constants: cells, depth weights, dip limits
  PointCells pc;
  pc.ok = false;
  float tan[4] = {0.f, 0.f, 0.f, 0.f}, acc = 0.f, cmp = 0.f;
  // Every operation below that feeds an index, a mask or the image is an
  // explicit IEEE operation (fused multiply-adds written out), so that the
  // FP32 C restatement in the oracle computes the same bits from the same
  // panels.
  const float z = __fmul_rn((float)izi, a.dzi);
  if (live) {
    const size_t k = (size_t)ixi * a.nzi + izi;
#pragma unroll
    for (int j = 0; j < 4; ++j) tan[j] = dips[j * a.nxz + k];
    acc = img[(size_t)ixb * a.nzi + izi];
    if (comp) cmp = comp[(size_t)ixb * a.nzi + izi];
    setup_cells(pc, ixi, z, a, dt, dq);
  }
  const bool act = live && pc.ok;
  const float tz = a.taperzone;
  // tan -/+ tz (1 + tan^2): the limits widened by the taper zone
  DipLimits d;
  d.x1 = tan[0], d.x2 = tan[1], d.y1 = tan[2], d.y2 = tan[3];
  d.x1c = __fsub_rn(d.x1, __fmul_rn(tz, __fmaf_rn(d.x1, d.x1, 1.0f)));
  d.x2c = __fadd_rn(d.x2, __fmul_rn(tz, __fmaf_rn(d.x2, d.x2, 1.0f)));
  d.y1c = __fsub_rn(d.y1, __fmul_rn(tz, __fmaf_rn(d.y1, d.y1, 1.0f)));
  d.y2c = __fadd_rn(d.y2, __fmul_rn(tz, __fmaf_rn(d.y2, d.y2, 1.0f)));
  d.wide = d.x1 > d.x1c && d.x2 < d.x2c && d.y1 > d.y1c && d.y2 < d.y2c;
  const float z2 = __fmul_rn(z, z);
  const float x = __fmul_rn((float)ixi, a.dxi);
  const float inv_dt1 = __fdiv_rn(1.0f, a.dt1), inv_dts = __fdiv_rn(1.0f, a.dtstar);
  const size_t pstride = (size_t)a.nbins * a.nt;
  const int plane = a.nxi1 * a.nzi1;

  tile_limits(act, d.x1c, d.x2c, d.y1c, d.y2c, s_red);
  {
    const float big = 3.0e38f;
    const bool wide = (int64_t)pc.nxs * pc.nys * plane >= (1ll << 30);
    block_min<8>(act ? (float)pc.cA : big, s_red, 8);
    block_min<8>(act ? -(float)pc.cA : big, s_red, 9);
    block_min<8>(act ? (float)pc.cB : big, s_red, 10);
    block_min<8>(act ? -(float)pc.cB : big, s_red, 11);
    block_min<8>(act ? (pc.same && !wide ? 0.0f : -1.0f) : big, s_red, 12);
    const unsigned on = __ballot_sync(0xffffffffu, act);
    if (lane == 0 && sums) s_col[lx] = __popc(on);
  }
  const int col_lo = ixb0 + a.ixstart, col_hi = min(ixb0 + TX, a.nxb) - 1 + a.ixstart;
  const int nrow = min(32, a.nzi - iz0);
  __syncthreads();
  bool uni;
  {
    float r[5];
#pragma unroll
    for (int k = 0; k < 5; ++k) {
      r[k] = s_red[8 + k][0];
#pragma unroll
      for (int w = 1; w < 8; ++w) r[k] = fminf(r[k], s_red[8 + k][w]);
    }
    uni = tq && r[0] == -r[1] && r[2] == -r[3] && r[4] == 0.0f;
  }
  if (tid == 0)
    s_box = tile_box(s_red, col_lo * a.dxi, col_hi * a.dxi, iz0 * a.dzi,
                     (iz0 + nrow - 1) * a.dzi);
  if (uni && act && atomicCAS(&s_tgw, -1, tid) == -1)
    s_tg = TileGrid{pc.xc, pc.rdx, pc.rdy, pc.hx, pc.hy, pc.nxs, pc.nys};
  __syncthreads();
  int tsx = 0, tsy = 0;
  const float4 *tab = tq;
  if (uni && act) {
    tsx = s_tg.nxs > 1 ? plane : 0, tsy = s_tg.nys > 1 ? s_tg.nxs * plane : 0;
    tab = tq + pc.tA + pc.offA;
  }
  // (t, t*) at the point from the tile's surface grid
  auto lookup_uni = [&](int off, float wx, float wy, float &t, float &q) {
    ulonglong2 n[4];
    load_nodes(tab + off, tsx, tsy, n);
    f2 v[2];
    bilin_tq(n, f2_dup(wx), f2_dup(wy), v);
    const float2 A = f2_unpack(v[0]), B = f2_unpack(v[1]);
    t = lerp(A.x, B.x, pc.c2);
    q = lerp(A.y, B.y, pc.c2);
  };
  // source terms are reused while consecutive traces share a source
  float last_sx = NAN, last_sy = NAN, ts = 0.f, qs = 0.f, dsx = 0.f, ds = 0.f, rs = 0.f;
  bool s_ok = false;
  unsigned cnt = 0, cimg = 0;

  auto keep = [&](int i, int4 &r, float4 &g, float2 &h) {
    h = make_float2(0.0f, 0.0f);
    const int4 q0 = *reinterpret_cast<const int4 *>(ints + (size_t)i * kGateInts);
    if (q0.x != kAccepted) return false;
    const int4 q1 = *reinterpret_cast<const int4 *>(ints + (size_t)i * kGateInts + 4);
    const int lo = max(q1.x, col_lo), hi = min(q1.y, col_hi);
    if (lo > hi || q1.w >= iz0 + nrow) return false;
    g = *reinterpret_cast<const float4 *>(geom + (size_t)i * kGateF);
    // record: trace, columns, first depth, table offset
    r = make_int4(i, (lo - col_lo) | (hi - col_lo) << 8, q1.w, 0);
    if (!uni) return true;
    const float2 sp = make_float2(g.x, g.y), gp = make_float2(g.z, g.w);
    if (!tile_covers(s_tg, sp) || !tile_covers(s_tg, gp)) return false;
    // point-traces: the active points (the first rows of each column) from q1.w on
    for (int c = lo - col_lo; c <= hi - col_lo; ++c) cnt += max(0, s_col[c] - max(0, q1.w - iz0));
    surface_weights(s_tg, gp.x, gp.y, plane, r.w, h.x, h.y);
    return tile_keep(sp, gp, s_box);
  };
  auto eval = [&](int k, float &val) {
    const int4 r = sm.rec[k];
    const float4 gm = sm.geo[k];
    if (lx < (r.y & 0xFF) || lx > r.y >> 8 || izi < r.z) return false;
    float tg, qg;
    if (gm.x != last_sx || gm.y != last_sy) {
      last_sx = gm.x;
      last_sy = gm.y;
      if (uni) {
        int off;
        float wx, wy;
        surface_weights(s_tg, gm.x, gm.y, plane, off, wx, wy);
        lookup_uni(off, wx, wy, ts, qs);
        s_ok = true;
      } else {
        s_ok = lookup_tq(pc, dt, ttt, dq, qqq, tq, a.nxi1, a.nzi1, gm.x, gm.y, ts, qs);
      }
      dsx = __fsub_rn(gm.x, x);
      ds = __fsqrt_rn(__fmaf_rn(dsx, dsx, __fmaf_rn(gm.y, gm.y, z2)));
      rs = __fdiv_rn(1.0f, ds);
    }
    if (!uni) {
      if (!s_ok) return false;
      if (!lookup_tq(pc, dt, ttt, dq, qqq, tq, a.nxi1, a.nzi1, gm.z, gm.w, tg, qg)) return false;
      ++cnt;  // a point-trace: in the aperture, table values at both ends
    }
    // ray directions and dip taper (src/q-psdm.cu:2303-2340)
    const float dgx = __fsub_rn(gm.z, x);
    const float dg = __fsqrt_rn(__fmaf_rn(dgx, dgx, __fmaf_rn(gm.w, gm.w, z2)));
    const float rg2 = __frcp_rn(dg);
    const float ux = __fmaf_rn(dsx, rs, __fmul_rn(dgx, rg2));
    const float uy = __fmaf_rn(gm.y, rs, __fmul_rn(gm.w, rg2));
    const float uz = __fmul_rn(z, __fadd_rn(rs, rg2));
    float w;
    if (!dip_taper(ux, uy, uz, d, w)) return false;
    if (uni) {
      const float2 h = sm.wgt[k];
      lookup_uni(r.w, h.x, h.y, tg, qg);
    }
    // time and t* picks (src/q-psdm.cu:2354-2357)
    const float t = __fadd_rn(ts, tg);
    const float ft = __fmul_rn(t, inv_dt1);
    const int it1 = (int)ft;
    if (!(it1 > 0 && it1 < a.nt - 1)) return false;  // (it1 is INT_MAX past its range)
    ++cimg;
    const float wt = __fsub_rn(ft, (float)it1);
    const float fb = fminf(fmaxf(__fmul_rn(__fadd_rn(qs, qg), inv_dts), 0.0f),
                           (float)(a.nbins - 1));
    const int b0 = min((int)fb, a.nbins - 2);
    const float wb = __fsub_rn(fb, (float)b0);
    const T *pp = panels + (size_t)r.x * pstride + (size_t)b0 * a.nt + it1;
    const float p00 = ld_sample<T>(pp), p01 = ld_sample<T>(pp + 1);
    const float p10 = ld_sample<T>(pp + a.nt), p11 = ld_sample<T>(pp + a.nt + 1);
    float smp = lerp(lerp(p00, p01, wt), lerp(p10, p11, wt), wb);
    if (std::is_same<T, __half>::value) smp = __fmul_rn(smp, __ldg(pscale + r.x));
    // amplitude weight (src/q-psdm.cu:2366-2374): w v (r + 1/r),
    // r = (ds/dg)^3 tg/ts, v = 100 / t^2 (10^4 below 0.1 s)
    const float v = t > 0.1f ? __fdiv_rn(100.0f, __fmul_rn(t, t)) : 10000.0f;
    const float dr = __fmul_rn(ds, rg2);
    const float rr = __fmul_rn(__fmul_rn(__fmul_rn(dr, dr), dr), __fdiv_rn(tg, ts));
    val = __fmul_rn(__fmul_rn(__fmul_rn(w, __fadd_rn(rr, __frcp_rn(rr))), v), smp);
    return true;
  };
  ordered_walk<SPLIT>(sm, ntr, act, keep, eval, [&](float val) {
    if (comp) {  // Kahan-compensated sum
      const float y = __fsub_rn(val, cmp);
      const float tt = __fadd_rn(acc, y);
      cmp = __fsub_rn(__fsub_rn(tt, acc), y);
      acc = tt;
    } else {
      acc = __fadd_rn(acc, val);
    }
  });
  if (live && sums) {
    img[(size_t)ixb * a.nzi + izi] = acc;
    if (comp) comp[(size_t)ixb * a.nzi + izi] = cmp;
  }
  if (npt) add_counts(npt, s_cnt, cnt, 0u, cimg);
}

// ---------------------------------------------------------------------------
// batched form
// ---------------------------------------------------------------------------
constexpr unsigned long long kNoKey = ~0ull;

// Receiver keys (accepted traces; position bits of the gate's relative
// coordinates), trace indices, and source-run flags from the raw headers.
__global__ void k_batch_keys(const uint8_t *__restrict__ rec, int rec_bytes, int be, int ntr,
                             const int *__restrict__ ints, const float *__restrict__ geom,
                             unsigned long long *__restrict__ key, int *__restrict__ val,
                             int *__restrict__ srcflag, int *__restrict__ naccepted) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  // accepted members of the batch (they sort first: rejected keys are the largest)
  const bool acc = i < ntr && ints[(size_t)i * kGateInts] == kAccepted;
  const unsigned ballot = __ballot_sync(0xffffffffu, acc);
  if ((threadIdx.x & 31) == 0 && ballot) atomicAdd(naccepted, __popc(ballot));
  if (i >= ntr) return;
  const uint8_t *r = rec + (size_t)i * rec_bytes;
  int flag = 1;
  if (i > 0) {
    const uint8_t *q = r - rec_bytes;
    flag = su_i32(r, kOffSx, be) != su_i32(q, kOffSx, be) ||
           su_i32(r, kOffSy, be) != su_i32(q, kOffSy, be);
  }
  srcflag[i] = flag;
  const bool ok = acc;
  const float gx = geom[(size_t)i * kGateF + 2], gy = geom[(size_t)i * kGateF + 3];
  key[i] = ok ? ((unsigned long long)__float_as_uint(gy) << 32) | __float_as_uint(gx) : kNoKey;
  val[i] = i;
}

// Receiver position of every receiver group (run of equal keys).
__global__ void k_batch_groups(const unsigned long long *__restrict__ ukey,
                               const int *__restrict__ nruns, float2 *__restrict__ grppos,
                               int ntr) {
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= ntr || g >= *nruns) return;
  const unsigned long long k = ukey[g];  // rejected traces (kNoKey) are never imaged
  grppos[g] = make_float2(__uint_as_float((unsigned)(k & 0xffffffffu)),
                          __uint_as_float((unsigned)(k >> 32)));
}

// The group of every sorted position: the last run whose first position is
// at or before it (off: exclusive prefix sums of the run lengths).
__global__ void k_batch_memgrp(const int *__restrict__ off, const int *__restrict__ nruns,
                               int *__restrict__ memgrp, int ntr) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= ntr) return;
  int lo = 0, hi = *nruns;  // off[lo] <= p < off[hi] (off[nruns] taken as ntr)
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (off[mid] <= p) lo = mid; else hi = mid;
  }
  memgrp[p] = lo;
}

// Member info per sorted position (trace, source, column range) and the
// position of every source run (the gate's double-precision arithmetic).
__global__ void k_batch_members(const uint8_t *__restrict__ rec, int rec_bytes, int be, int ntr,
                                const int *__restrict__ sval, const int *__restrict__ ints,
                                const int *__restrict__ sid, const int *__restrict__ srcflag,
                                double scaled, double fxi, double cyi,
                                const float *__restrict__ pscale, int4 *__restrict__ mem,
                                float2 *__restrict__ srcpos) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= ntr) return;
  const int j = sval[p];
  const int *q = ints + (size_t)j * kGateInts;
  // member record: trace, source slot (bits 0-23) with the exponent of the
  // trace's FP16 sample multiplier + 128 (bits 24-31), cdp range
  int e = 0;
  if (pscale && q[0] == kAccepted) e = min(max(ilogbf(pscale[j]), -126), 127);
  mem[p] = q[0] == kAccepted ? make_int4(j, (sid[j] - 1) | ((e + 128) << 24), q[4], q[5])
                             : make_int4(j, -1, 1, 0);
  if (srcflag[p]) {  // p as a trace index: first trace of a source run
    const uint8_t *r = rec + (size_t)p * rec_bytes;
    const double sx = __dmul_rn((double)su_i32(r, kOffSx, be), scaled);
    const double sy = __dmul_rn((double)su_i32(r, kOffSy, be), scaled);
    srcpos[sid[p] - 1] = make_float2(__double2float_rn(__dsub_rn(sx, fxi)),
                                     __double2float_rn(__dsub_rn(sy, cyi)));
  }
}

// Source terms kept per (source, point) in shared memory, as four float2
// planes [plane][source][point]: (T, t* / dtstar), (CS = ds^3 / ts, AZ),
// (PX1, PX2), (PY1, PY2), with A the unit vector from the point to the source
// and
//   PX1 = AX - tanx1c AZ, PX2 = tanx2c AZ - AX   (PY likewise with tany)
// so that the dip test of a (source, receiver) pair needs no division: for
// uz = AZ + AZg > 0, tanx1c < ux / uz < tanx2c is PX1 > tanx1c AZg - AXg and
// PX2 > AXg - tanx2c AZg (the receiver's thresholds, once per receiver).
// The differences PX1 - (tanx1c AZg - AXg) etc. are the pair's dip-test
// functions, which also give the dip taper.
enum { kMapTQ = 0, kMapCZ, kMapPX, kMapPY, kMapN };

// A tile whose members are split into parts: true on every thread of the CTA
// whose part is the last one written (every part's sums are then visible).
__device__ __forceinline__ bool last_part(int *done, int nsplit, int *s_flag) {
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) *s_flag = atomicAdd(done, 1);
  __syncthreads();
  if (*s_flag != nsplit - 1) return false;
  __threadfence();
  return true;
}
// A part's sum of a point, and its compensation behind it (compensated sums: a part
// rounded to one float would lose what the compensation had kept).
__device__ __forceinline__ void put_part(float *part, size_t nimg, int ipart, float acc, float cmp,
                                         bool comp) {
  if (comp) {
    part[2 * ipart * nimg] = acc;
    part[(2 * ipart + 1) * nimg] = cmp;
  } else {
    part[ipart * nimg] = acc;
  }
}
// Adds a point's nsplit partial sums to the image in order.  Compensated: a sum
// is s - c; parts are as large as the image, so the whole error of each addition
// is taken (Knuth's two-sum), where a step of the compensated sum would round
// the part minus c.
__device__ __forceinline__ void add_parts(float *img, float *comp, const float *part, size_t nimg,
                                          int nsplit) {
  float s = *img;
  if (!comp) {
    for (int i = 0; i < nsplit; ++i) s += __ldcg(part + i * nimg);
    *img = s;
    return;
  }
  float c = *comp;
  for (int i = 0; i < nsplit; ++i) {
    const float v = __ldcg(part + 2 * i * nimg), t = s + v, b = t - s;
    const float e = (s - (t - b)) + (v - b);
    c = (c - e) + __ldcg(part + (2 * i + 1) * nimg);
    s = t;
  }
  const float t = s - c;
  *img = t;
  *comp = (t - s) + c;
}

// Batched imaging.  A persistent CTA takes image tiles of TZ depths x TX
// cdps (one thread per point) from a counter.  Per tile and per chunk of sc
// sources: the source terms of every point in shared memory; then the
// members (traces in receiver order) in chunks of 32 x NT: the CTA keeps the
// members that pass the tile-level dip test (a bit mask), and every point
// runs over the kept members in order -- receiver terms once per receiver
// group, the members in blocks of U (the per-point aperture and dip tests,
// then the time/t* pick, weight and panel gathers).  Members dropped for the
// tile fail every point's dip test, so the image is that of running every
// member.  A point-trace is a pair in the trace's aperture whose source and
// receiver both have table values at the point: in a tile whose active
// points all read the same table cells (the usual case) one surface-grid
// test per member decides that for the whole tile, members outside the grid
// are dropped too, and a member dropped by the dip bound counts its
// in-aperture points; in any other tile every member goes to the points,
// which count for themselves.  nsplit > 1: an item of the queue is one of
// nsplit parts of a tile's members (small images have fewer tiles than the
// GPU has room for); a part leaves its sums in part[], and the part that
// finishes a tile last adds all of them to the image in order.
template <int TZ, int TX, int MB, int U, typename T>
__global__ void __launch_bounds__(TZ *TX, MB)
    k_image_batched(float *__restrict__ img, float *__restrict__ comp, PhysImageArgs a,
                    const float *__restrict__ dips, const int *__restrict__ memgrp,
                    const float2 *__restrict__ grppos, const int4 *__restrict__ mem,
                    const int *__restrict__ nmem_ptr,
                    const float2 *__restrict__ srcpos, const int *__restrict__ nsrc_ptr,
                    const qpsdm_ttt_desc *__restrict__ dt, const float *__restrict__ ttt,
                    const qpsdm_ttt_desc *__restrict__ dq, const float *__restrict__ qqq,
                    const float4 *__restrict__ tqp, const T *__restrict__ panels,
                    int *__restrict__ tile_ctr, int ntz, int ntx, int sc,
                    unsigned long long *npt, const int *__restrict__ tile_list,
                    const int *__restrict__ ntile_list, int nsplit, float *__restrict__ part,
                    int *__restrict__ tile_done) {
  constexpr int NT = TZ * TX, NW = NT / 32, MC = 32 * NT;
  static_assert(NT % 32 == 0, "whole warps");
  const int nmem_all = *nmem_ptr;  // the accepted members (sorted first)
  extern __shared__ float2 smap[];  // [kMapN][sc][NT]
  __shared__ unsigned s_mask[NT];   // kept members of the chunk, one bit each
  __shared__ int s_col[TX + 1];     // active points of the tile's columns (prefix sums)
  __shared__ float s_red[13][NW];
  __shared__ TileGrid s_tg;         // the tile's shared surface grid (uniform tiles)
  __shared__ int s_tgw;             // the thread that writes it
  __shared__ int s_tile, s_part;
  __shared__ unsigned long long s_cnt[3];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int lz = tid % TZ, lx = tid / TZ;
  const int nsrc = *nsrc_ptr;
  const float inv_dt1 = 1.0f / a.dt1, inv_dts = 1.0f / a.dtstar;
  const size_t pstride = (size_t)a.nbins * a.nt;
  unsigned cnt = 0, cdrop = 0, cimg = 0;
  for (;;) {
    __syncthreads();
    if (tid == 0) {
      // the next tile: from the counter, or the next of a list of tiles
      const int item = atomicAdd(tile_ctr, 1), q = item / nsplit;
      s_part = item - q * nsplit;
      s_tile = tile_list ? (q < *ntile_list ? tile_list[q] : ntz * ntx) : q;
      s_tgw = -1;
    }
    if (tid <= TX) s_col[tid] = 0;
    __syncthreads();
    const int tile = s_tile, ipart = s_part;
    if (tile >= ntz * ntx) break;
    // this item's members: chunks ipart, ipart + nsplit, ... of clen each
    const int clen = nsplit > 1 ? min(kSplitChunk, (nmem_all + nsplit - 1) / nsplit) : MC;
    const int iz0 = (tile % ntz) * TZ, ixb0 = (tile / ntz) * TX;
    const int izi = iz0 + lz;
    const int ixb = ixb0 + lx;
    const bool live = izi < a.nzi && ixb < a.nxb;
    const int ixi = ixb + a.ixstart;
    PointCells pc;
    pc.ok = false;
    float tanx1 = 0.f, tanx2 = 0.f, tany1 = 0.f, tany2 = 0.f, acc = 0.f, cmp = 0.f;
    const float z = izi * a.dzi;
    if (live) {
      const size_t k = (size_t)ixi * a.nzi + izi;
      tanx1 = dips[k];
      tanx2 = dips[a.nxz + k];
      tany1 = dips[2 * a.nxz + k];
      tany2 = dips[3 * a.nxz + k];
      if (nsplit == 1) {
        acc = img[(size_t)ixb * a.nzi + izi];
        if (comp) cmp = comp[(size_t)ixb * a.nzi + izi];
      }
      setup_cells(pc, ixi, z, a, dt, dq);
    }
    const bool act = live && pc.ok;
    const float tz = a.taperzone;
    const float tanx1c = tanx1 - tz * (1.0f + tanx1 * tanx1);
    const float tanx2c = tanx2 + tz * (1.0f + tanx2 * tanx2);
    const float tany1c = tany1 - tz * (1.0f + tany1 * tany1);
    const float tany2c = tany2 + tz * (1.0f + tany2 * tany2);
    // inverse taper-zone widths: the taper factor at a passing pair is
    // min(1, f / (w uz)) for the test function f of each limit, w = |tan - tanc|
    const float iwx1 = 1.0f / (tanx1 - tanx1c), iwx2 = 1.0f / (tanx2c - tanx2);
    const float iwy1 = 1.0f / (tany1 - tany1c), iwy2 = 1.0f / (tany2c - tany2);
    const float z2 = z * z;
    const float x = ixi * a.dxi;
    // the tile's box and dip-limit ranges over its active points
    {
      const float big = 3.0e38f;
      block_min<NW>(act ? tanx1c : big, s_red, 0);
      block_min<NW>(act ? -tanx1c : big, s_red, 1);
      block_min<NW>(act ? tanx2c : big, s_red, 2);
      block_min<NW>(act ? -tanx2c : big, s_red, 3);
      block_min<NW>(act ? tany1c : big, s_red, 4);
      block_min<NW>(act ? -tany1c : big, s_red, 5);
      block_min<NW>(act ? tany2c : big, s_red, 6);
      block_min<NW>(act ? -tany2c : big, s_red, 7);
      // the table cells of the tile's points (exact in float: cells < 2^24)
      block_min<NW>(act ? (float)pc.cA : big, s_red, 8);
      block_min<NW>(act ? -(float)pc.cA : big, s_red, 9);
      block_min<NW>(act ? (float)pc.cB : big, s_red, 10);
      block_min<NW>(act ? -(float)pc.cB : big, s_red, 11);
      block_min<NW>(act ? (pc.same ? 0.0f : -1.0f) : big, s_red, 12);
      if (act) atomicAdd(&s_col[lx + 1], 1);
    }
    __syncthreads();
    if (tid == 0)
      for (int c = 1; c <= TX; ++c) s_col[c] += s_col[c - 1];
    TileBox box;
    bool uni;  // every active point reads the same cells on one surface grid
    {
      float r[13];
#pragma unroll
      for (int k = 0; k < 13; ++k) {
        r[k] = s_red[k][0];
#pragma unroll
        for (int w = 1; w < NW; ++w) r[k] = fminf(r[k], s_red[k][w]);
      }
      box.t1lo = r[0], box.t1hi = -r[1], box.t2lo = r[2], box.t2hi = -r[3];
      box.u1lo = r[4], box.u1hi = -r[5], box.u2lo = r[6], box.u2hi = -r[7];
      float tmax = 1.0f;
#pragma unroll
      for (int k = 0; k < 8; ++k) tmax = fmaxf(tmax, fabsf(r[k]));
      box.margin = -1e-4f * tmax;
      const int ncol = min(TX, a.nxb - ixb0), nrow = min(TZ, a.nzi - iz0);
      box.x0 = (ixb0 + a.ixstart) * a.dxi;
      box.x1 = (ixb0 + a.ixstart + ncol - 1) * a.dxi;
      box.z0 = iz0 * a.dzi;
      box.z1 = (iz0 + nrow - 1) * a.dzi;
      uni = r[8] == -r[9] && r[10] == -r[11] && r[12] == 0.0f;
      if (uni && act && atomicCAS(&s_tgw, -1, tid) == -1)
        s_tg = TileGrid{pc.xc, pc.rdx, pc.rdy, pc.hx, pc.hy, pc.nxs, pc.nys};
    }
    __syncthreads();  // s_col and s_tg complete
    if (s_col[TX] == 0) continue;  // no active point in the tile
    const int ixi_lo = ixb0 + a.ixstart, ixi_hi = ixi_lo + min(TX, a.nxb - ixb0) - 1;

    for (int s0 = 0; s0 < nsrc; s0 += sc) {
      const int ns = min(sc, nsrc - s0);
      // source terms of this chunk for this thread's point
      for (int s = 0; s < ns && act; ++s) {
        const float2 sp = srcpos[s0 + s];
        float ts, qs;
        float2 *m = smap + (size_t)s * NT + tid;
        if (!lookup_tq(pc, dt, ttt, dq, qqq, tqp, a.nxi1, a.nzi1, sp.x, sp.y, ts, qs)) {
          // no table value: NaN fails every member's dip test
          m[kMapTQ * sc * NT] = make_float2(NAN, 0.0f);
          m[kMapCZ * sc * NT] = make_float2(0.0f, NAN);
          m[kMapPX * sc * NT] = make_float2(NAN, NAN);
          m[kMapPY * sc * NT] = make_float2(NAN, NAN);
          continue;
        }
        const float dsx = sp.x - x;
        const float ds = sqrtf(dsx * dsx + sp.y * sp.y + z2);
        const float rds = __fdividef(1.0f, ds);
        const float ax = dsx * rds, ay = sp.y * rds, az = z * rds;
        m[kMapTQ * sc * NT] = make_float2(ts, qs * inv_dts);  // t* in bins
        // source factor of (ds/dg)^3 tg/ts
        m[kMapCZ * sc * NT] = make_float2(__fdividef(ds * ds * ds, ts), az);
        m[kMapPX * sc * NT] = make_float2(fmaf(-tanx1c, az, ax), fmaf(tanx2c, az, -ax));
        m[kMapPY * sc * NT] = make_float2(fmaf(-tany1c, az, ay), fmaf(tany2c, az, -ay));
      }
      for (int pc0 = ipart * clen; pc0 < nmem_all; pc0 += nsplit * clen) {
        const int nmem = min(pc0 + clen, nmem_all);
        // the chunk's members kept for this tile (warp w, round k: word k NW + w)
#pragma unroll 4
        for (int k = 0; k < MC / NT; ++k) {
          const int wi = k * NW + warp;
          const int p = pc0 + 32 * wi + lane;
          bool keep = false;
          if (p < nmem) {
            const int4 mi = __ldg(mem + p);
            const int sl = (mi.y & 0xFFFFFF) - s0;
            const int lo = max(mi.z, ixi_lo), hi = min(mi.w, ixi_hi);
            if (sl >= 0 && sl < ns && lo <= hi) {
              if (uni) {
                const float2 sp = __ldg(srcpos + s0 + sl), gp = __ldg(grppos + __ldg(memgrp + p));
                const bool cov = tile_covers(s_tg, sp) && tile_covers(s_tg, gp);
                keep = cov && tile_keep(sp, gp, box);
                // dropped by the dip bound: its in-aperture points still count
                if (cov && !keep) cdrop += s_col[hi - ixi_lo + 1] - s_col[lo - ixi_lo];
              } else {
                keep = true;  // several cells in the tile: every point decides alone
              }
            }
          }
          const unsigned bits = __ballot_sync(0xffffffffu, keep);
          if (lane == 0) s_mask[wi] = bits;
        }
        __syncthreads();
        if (act) {
          // kept members in order: word w of the mask, remaining bits mw
          int w = 0;
          unsigned mw = s_mask[0];
          auto next = [&]() -> int {
            while (mw == 0) {
              if (++w >= NT) return -1;
              mw = s_mask[w];
            }
            const int b = __ffs(mw) - 1;
            mw &= mw - 1;
            return pc0 + 32 * w + b;
          };
          int nxt = next();
          int gn = nxt >= 0 ? __ldg(memgrp + nxt) : -1;
          int cur = -1;
          float agx = 0.f, agy = 0.f, agz = 0.f, qx1 = 0.f, qx2 = 0.f, qy1 = 0.f, qy2 = 0.f;
          float tg = 0.f, qg = 0.f, gfac = 0.f;
          bool rok = false;  // the current receiver has table values at this point
          while (nxt >= 0) {
            const int g = gn;
            if (g != cur) {
              cur = g;
              // receiver terms, once per receiver position
              const float2 gp = __ldg(grppos + g);
              rok = lookup_tq(pc, dt, ttt, dq, qqq, tqp, a.nxi1, a.nzi1, gp.x, gp.y, tg, qg);
              const float dgx = gp.x - x;
              const float rdg = rsqrtf(dgx * dgx + gp.y * gp.y + z2);  // 1 / dg
              agx = dgx * rdg, agy = gp.y * rdg, agz = z * rdg;
              // dip-test thresholds of this receiver (NaN: no table value,
              // every member fails)
              qx1 = rok ? fmaf(tanx1c, agz, -agx) : NAN;
              qx2 = fmaf(-tanx2c, agz, agx);
              qy1 = fmaf(tany1c, agz, -agy);
              qy2 = fmaf(-tany2c, agz, agy);
              gfac = tg * rdg * rdg * rdg;  // receiver factor of (ds/dg)^3 tg/ts
              qg *= inv_dts;                // t* in bins
            }
            // up to U kept members of this receiver group
            int pm[U];
            pm[0] = nxt;
            nxt = next();
            gn = nxt >= 0 ? __ldg(memgrp + nxt) : -1;
#pragma unroll
            for (int u = 1; u < U; ++u) {
              if (gn == g) {
                pm[u] = nxt;
                nxt = next();
                gn = nxt >= 0 ? __ldg(memgrp + nxt) : -1;
              } else {
                pm[u] = -1;
              }
            }
            // Phase 1, without branches, for all U: the member record, the
            // aperture check (counted), the source direction and the dip
            // test.  Phase 2: time/t* pick and weight of the members that
            // passed.  Then all panel gathers, then the sums (in member
            // order), so that U members' loads are in flight together.
            int4 mi[U];
#pragma unroll
            for (int u = 0; u < U; ++u)
              mi[u] = pm[u] >= 0 ? __ldg(mem + pm[u]) : make_int4(0, -1, 1, 0);
            bool on[U];
            int slv[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
              const int sl = (mi[u].y & 0xFFFFFF) - s0;
              const bool inr = (unsigned)sl < (unsigned)ns && ixi >= mi[u].z && ixi <= mi[u].w;
              slv[u] = inr ? sl : 0;
              const float2 *m = smap + (size_t)slv[u] * NT + tid;
              const float2 px = m[kMapPX * sc * NT], py = m[kMapPY * sc * NT];
              // source terms are NaN where the source has no table value
              cnt += (inr && rok && px.x == px.x) ? 1u : 0u;
              on[u] = inr && px.x > qx1 && px.y > qx2 && py.x > qy1 && py.y > qy2;
            }
            const T *pp[U];
            float fwt[U], fwb[U], fac[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
              pp[u] = panels;
              fwt[u] = fwb[u] = fac[u] = 0.0f;
              if (!on[u]) continue;
              on[u] = false;
              const float2 *m = smap + (size_t)slv[u] * NT + tid;
              const float2 tq = m[kMapTQ * sc * NT], cz = m[kMapCZ * sc * NT];
              const float2 px = m[kMapPX * sc * NT], py = m[kMapPY * sc * NT];
              const float ts = tq.x;
              // dip taper from the pair's test functions (ux - tanx1c uz and
              // the like, all > 0 here): (tanx - tanx1c) / (tanx1 - tanx1c) =
              // (ux - tanx1c uz) / ((tanx1 - tanx1c) uz) below tanx1, likewise
              // at the other three limits; of the two limits of an axis at
              // most one taper is active, so each axis takes the smaller ratio
              const float ruz = __fdividef(1.0f, cz.y + agz);
              const float ex = fminf((px.x - qx1) * iwx1, (px.y - qx2) * iwx2);
              const float ey = fminf((py.x - qy1) * iwy1, (py.y - qy2) * iwy2);
              const float wt = fminf(1.0f, ex * ruz) * fminf(1.0f, ey * ruz);
              const float t = ts + tg;
              const float ft = t * inv_dt1;
              const int it1 = (int)ft;
              if (!(it1 > 0 && it1 < a.nt - 1)) continue;  // (it1: INT_MAX past its range)
              const float fb = fminf(fmaxf(tq.y + qg, 0.0f), (float)(a.nbins - 1));
              const int b0 = min((int)fb, a.nbins - 2);
              fwt[u] = ft - (float)it1;
              fwb[u] = fb - (float)b0;
              pp[u] = panels + (size_t)mi[u].x * pstride + (unsigned)(b0 * a.nt + it1);
              // w v (r + 1/r), v = 100 / t^2 (10^4 below 0.1 s), with one
              // reciprocal: w (r^2 + 1) * 100 / (r t^2)
              const float r = cz.x * gfac;
              const bool far = t > 0.1f;
              fac[u] = wt * fmaf(r, r, 1.0f) *
                       __fdividef(far ? 100.0f : 10000.0f, far ? r * t * t : r);
              if (std::is_same<T, __half>::value)  // 2^e from the record's exponent bits
                fac[u] *= __int_as_float((int)((((unsigned)mi[u].y >> 24) - 1u) << 23));
              on[u] = true;
              ++cimg;
            }
            float smp[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
              smp[u] = 0.0f;
              if (on[u]) {
                const T *q = pp[u];
                const float p00 = ld_sample<T>(q), p01 = ld_sample<T>(q + 1);
                const float p10 = ld_sample<T>(q + a.nt), p11 = ld_sample<T>(q + a.nt + 1);
                const float s0v = p00 + fwt[u] * (p01 - p00), s1v = p10 + fwt[u] * (p11 - p10);
                smp[u] = s0v + fwb[u] * (s1v - s0v);
              }
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
              if (!on[u]) continue;
              const float val = fac[u] * smp[u];
              if (comp) {
                const float y = val - cmp;
                const float tt = acc + y;
                cmp = (tt - acc) - y;
                acc = tt;
              } else {
                acc += val;
              }
            }
          }
        }
        __syncthreads();  // the mask is rewritten by the next chunk
      }
    }
    const size_t o = (size_t)ixb * a.nzi + izi;
    if (nsplit == 1) {
      if (live) {
        img[o] = acc;
        if (comp) comp[o] = cmp;
      }
      continue;
    }
    const size_t nimg = (size_t)a.nxb * a.nzi;
    if (live) put_part(part + o, nimg, ipart, acc, cmp, comp);
    if (!last_part(tile_done + tile, nsplit, &s_tile)) continue;
    if (live) add_parts(img + o, comp ? comp + o : nullptr, part + o, nimg, nsplit);
  }
  if (npt) add_counts(npt, s_cnt, cnt + cdrop, cdrop, cimg);
}

__device__ __forceinline__ float rsqrt_fast(float x) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float rcp_fast(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Batched imaging, fast form: the same sums as k_image_batched for the tiles
// whose active points all read the same table cells of paired (t, t*)
// tables (with the tables' x-cells and depth cells aligned to the tile shape,
// every tile); any other tile is appended to defer[] (*ndefer of them) and
// left to k_image_batched.
//
// A thread holds two neighbouring depths of one cdp, and every FP32 operation
// of the walk runs on both in one f32x2 instruction; minima, reciprocals,
// comparisons and panel loads stay scalar.  The kernel is bound by issued
// instructions, and the two depths share what does not depend on depth: the
// member record, the range test, the table nodes of the receiver (when both
// depths lie between the same depth nodes: four pair loads and the bilinear
// surface interpolation at two nodes serve both), the horizontal part of the
// ray.  Integer parts (the time sample and the t* bin) come from adding 2^23
// towards zero, which leaves floor(x) in the low mantissa bits: no conversion
// instructions, whose unit runs at an eighth of the FP32 rate.
//
// The chunk's kept members are compacted in member order into shared memory:
// a record {trace, source slot | new receiver | column bits, table offset,
// 100 x FP16 scale} and {receiver position, surface weights}, so that every
// point reads broadcast records and no point recomputes what is the same for
// the tile.  Point-traces are counted per member in the keep pass (coverage
// is a tile-level test).  Source terms are four float4 planes per (source,
// pair of points), each holding two terms of both points: (PX1, PX2),
// (PY1, PY2), (T, t* / dtstar), (CS = ds^3 / ts, AZ).  One reciprocal per
// point-trace: inv = 1 / (uz r tt) gives both the taper's 1 / uz (r tt inv)
// and the weight's 1 / (r tt) (uz inv), tt = t^2 (0.01 below 0.1 s).  Every
// value that decides a pair -- the dip-test functions, t, t / dt1 -- is the
// same IEEE operation as in k_image_batched.
//
// Measured, image kernels of a brick of four 512 x 400 lines of 18,432 traces
// (5.8e8 kept, 4.5e8 imaged pairs a line): 21.3 ms with one point per thread
// and two members per instruction, 11.4 ms with this walk and split parts; a
// line alone is 3.1 ms, 229 warp instructions per member and 64 points, issue
// active 62 %, stalls long scoreboard (table nodes, panel samples) first.
// Loading the next receiver's nodes ahead (16 more registers, 16 warps) and
// two members per block were slower.
//
// nsplit: as in k_image_batched.
constexpr int kNewGroup = 0x100;
template <int TZ, int TX, int MB, int U, int MW, typename T>
__global__ void __launch_bounds__(TZ *TX / 2, MB)
    k_image_batched_fast(float *__restrict__ img, float *__restrict__ comp, PhysImageArgs a,
                         const float *__restrict__ dips, const int *__restrict__ memgrp,
                         const float2 *__restrict__ grppos, const int4 *__restrict__ mem,
                         const int *__restrict__ nmem_ptr,
                         const float2 *__restrict__ srcpos, const int *__restrict__ nsrc_ptr,
                         const qpsdm_ttt_desc *__restrict__ dt,
                         const qpsdm_ttt_desc *__restrict__ dq,
                         const float4 *__restrict__ tqp, const T *__restrict__ panels,
                         int *__restrict__ tile_ctr, int ntz, int ntx, int sc,
                         unsigned long long *npt, int *__restrict__ defer,
                         int *__restrict__ ndefer, int nsplit, float *__restrict__ part,
                         int *__restrict__ tile_done) {
  constexpr int NT = TZ * TX / 2, NW = NT / 32, MC = 32 * MW, HZ = TZ / 2;
  static_assert(NT % 32 == 0 && MW % NW == 0 && TX <= 16, "whole warps, whole words per warp");
  const int nmem_all = *nmem_ptr;
  extern __shared__ float4 smap4[];  // [4][sc][NT]
  __shared__ int4 s_rec[MC + U];     // the chunk's kept members, in member order
  __shared__ float4 s_geo[MC];       // their receivers: x, y, surface weights
  __shared__ unsigned s_mask[MW];    // kept members of the chunk, one bit each
  __shared__ int s_wpos[MW + 1];     // kept members before word w (s_wpos[MW]: all)
  __shared__ int s_col[TX + 1];      // active points of the tile's columns (prefix sums)
  __shared__ float s_red[14][NW];
  __shared__ TileGrid s_tg;
  __shared__ TileBox s_box;  // the tile's box and dip-limit ranges (keep pass only)
  __shared__ int64_t s_base;
  __shared__ int s_tgw;
  __shared__ int s_tile;
  __shared__ unsigned long long s_cnt[3];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int lz = 2 * (tid % HZ), lx = tid / HZ;
  const int nsrc = *nsrc_ptr;
  const float inv_dt1 = 1.0f / a.dt1, inv_dts = 1.0f / a.dtstar;
  // largest t* bin coordinate whose bin has a right neighbour
  const float fb_max = __int_as_float(__float_as_int((float)(a.nbins - 1)) - 1);
  const unsigned idx0 = 0x4B000000u * (unsigned)(a.nt + 1);  // 2^23's bits, of both integer parts
  const unsigned pstride = (unsigned)a.nbins * a.nt;
  const int splane = sc * NT;
  unsigned cnt = 0, cdrop = 0, cimg = 0;
  for (;;) {
    __syncthreads();
    if (tid == 0) {
      s_tile = atomicAdd(tile_ctr, 1);
      s_tgw = -1;
    }
    if (tid <= TX) s_col[tid] = 0;
    __syncthreads();
    const int item = s_tile;
    if (item >= ntz * ntx * nsplit) break;
    const int tile = item / nsplit, ipart = item - tile * nsplit;
    // this item's members: chunks ipart, ipart + nsplit, ... of clen each
    const int clen = nsplit > 1 ? min(kSplitChunk, (nmem_all + nsplit - 1) / nsplit) : MC;
    const int iz0 = (tile % ntz) * TZ, ixb0 = (tile / ntz) * TX;
    const int izi = iz0 + lz;
    const int ixb = ixb0 + lx;
    const int ixi = ixb + a.ixstart;
    const float x = ixi * a.dxi;
    bool live[2], act[2];
    int off0, off1;
    float zv[2], c2v[2], lim[4][2], iwv[4][2], accv[2], cmpv[2];
    {
      PointCells pc[2];
      float tc[4][2];
#pragma unroll
      for (int p = 0; p < 2; ++p) {
        live[p] = izi + p < a.nzi && ixb < a.nxb;
        pc[p].ok = false;
        zv[p] = (izi + p) * a.dzi;
        accv[p] = cmpv[p] = 0.0f;
        float tan[4] = {0.f, 0.f, 0.f, 0.f};
        if (live[p]) {
          const size_t k = (size_t)ixi * a.nzi + izi + p;
#pragma unroll
          for (int j = 0; j < 4; ++j) tan[j] = dips[j * a.nxz + k];
          if (nsplit == 1) {
            accv[p] = img[(size_t)ixb * a.nzi + izi + p];
            if (comp) cmpv[p] = comp[(size_t)ixb * a.nzi + izi + p];
          }
          setup_cells(pc[p], ixi, zv[p], a, dt, dq);
        }
        act[p] = live[p] && pc[p].ok;
        const float tz = a.taperzone;
        tc[0][p] = tan[0] - tz * (1.0f + tan[0] * tan[0]);
        tc[1][p] = tan[1] + tz * (1.0f + tan[1] * tan[1]);
        tc[2][p] = tan[2] - tz * (1.0f + tan[2] * tan[2]);
        tc[3][p] = tan[3] + tz * (1.0f + tan[3] * tan[3]);
        // inverse taper-zone widths: the taper factor at a passing pair is
        // min(1, f / (w uz)) for the test function f of each limit, w = |tan - tanc|
        iwv[0][p] = 1.0f / (tan[0] - tc[0][p]), iwv[1][p] = 1.0f / (tc[1][p] - tan[1]);
        iwv[2][p] = 1.0f / (tan[2] - tc[2][p]), iwv[3][p] = 1.0f / (tc[3][p] - tan[3]);
        // a point without table values fails every dip test
#pragma unroll
        for (int j = 0; j < 4; ++j) lim[j][p] = act[p] ? tc[j][p] : NAN;
      }
      if (act[0] && !act[1]) pc[1] = pc[0];
      off0 = pc[0].offA, off1 = pc[1].offA;
      c2v[0] = pc[0].c2, c2v[1] = pc[1].c2;
      const float big = 3.0e38f;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        block_min<NW>(fminf(act[0] ? tc[j][0] : big, act[1] ? tc[j][1] : big), s_red, 2 * j);
        block_min<NW>(fminf(act[0] ? -tc[j][0] : big, act[1] ? -tc[j][1] : big), s_red, 2 * j + 1);
      }
      // the table cells of the tile's points (exact in float: cells < 2^24)
      float cAl = big, cAh = big, cBl = big, cBh = big, same = big, apart = big;
#pragma unroll
      for (int p = 0; p < 2; ++p)
        if (act[p]) {
          cAl = fminf(cAl, (float)pc[p].cA), cAh = fminf(cAh, -(float)pc[p].cA);
          cBl = fminf(cBl, (float)pc[p].cB), cBh = fminf(cBh, -(float)pc[p].cB);
          const bool wide = (int64_t)pc[p].nxs * pc[p].nys * a.nxi1 * a.nzi1 >= (1ll << 30);
          same = fminf(same, pc[p].same && !wide ? 0.0f : -1.0f);
        }
      if (act[0]) apart = off0 == off1 ? 0.0f : -1.0f;
      block_min<NW>(cAl, s_red, 8);
      block_min<NW>(cAh, s_red, 9);
      block_min<NW>(cBl, s_red, 10);
      block_min<NW>(cBh, s_red, 11);
      block_min<NW>(same, s_red, 12);
      block_min<NW>(apart, s_red, 13);
      if (act[0]) {
        atomicAdd(&s_col[lx + 1], act[1] ? 2 : 1);
        if (atomicCAS(&s_tgw, -1, tid) == -1) {
          s_tg = TileGrid{pc[0].xc, pc[0].rdx, pc[0].rdy, pc[0].hx, pc[0].hy, pc[0].nxs,
                          pc[0].nys};
          s_base = pc[0].tA;
        }
      }
    }
    __syncthreads();
    if (tid == 0)
      for (int c = 1; c <= TX; ++c) s_col[c] += s_col[c - 1];
    bool uni, shared_nodes;
    {
      TileBox box;
      float r[14];
#pragma unroll
      for (int k = 0; k < 14; ++k) {
        r[k] = s_red[k][0];
#pragma unroll
        for (int w = 1; w < NW; ++w) r[k] = fminf(r[k], s_red[k][w]);
      }
      box.t1lo = r[0], box.t1hi = -r[1], box.t2lo = r[2], box.t2hi = -r[3];
      box.u1lo = r[4], box.u1hi = -r[5], box.u2lo = r[6], box.u2hi = -r[7];
      float tmax = 1.0f;
#pragma unroll
      for (int k = 0; k < 8; ++k) tmax = fmaxf(tmax, fabsf(r[k]));
      box.margin = -1e-4f * tmax;
      const int ncol = min(TX, a.nxb - ixb0), nrow = min(TZ, a.nzi - iz0);
      box.x0 = (ixb0 + a.ixstart) * a.dxi;
      box.x1 = (ixb0 + a.ixstart + ncol - 1) * a.dxi;
      box.z0 = iz0 * a.dzi;
      box.z1 = (iz0 + nrow - 1) * a.dzi;
      uni = r[8] == -r[9] && r[10] == -r[11] && r[12] == 0.0f;
      shared_nodes = r[13] == 0.0f;
      if (tid == 0) s_box = box;
    }
    __syncthreads();
    if (s_col[TX] == 0) continue;
    if (!uni) {  // left to k_image_batched
      if (tid == 0 && ipart == 0) defer[atomicAdd(ndefer, 1)] = tile;
      continue;
    }
    const int ixi_lo = ixb0 + a.ixstart, ixi_hi = ixi_lo + min(TX, a.nxb - ixb0) - 1;
    const int plane = a.nxi1 * a.nzi1;
    const int tsx = s_tg.nxs > 1 ? plane : 0, tsy = s_tg.nys > 1 ? s_tg.nxs * plane : 0;
    const float4 *const tab0 = tqp + s_base + off0, *const tab1 = tqp + s_base + off1;
    // (t, t*) of both points for a surface position
    auto lookup = [&](int off, float wx, float wy, unsigned long long &t, unsigned long long &q) {
      const unsigned long long wx2 = f2_dup(wx), wy2 = f2_dup(wy);
      ulonglong2 n[4];
      f2 v0[2], v1[2];
      load_nodes(tab0 + off, tsx, tsy, n);
      bilin_tq(n, wx2, wy2, v0);
      v1[0] = v0[0], v1[1] = v0[1];
      if (!shared_nodes) {
        load_nodes(tab1 + off, tsx, tsy, n);
        bilin_tq(n, wx2, wy2, v1);
      }
      const float2 A0 = f2_unpack(v0[0]), B0 = f2_unpack(v0[1]);
      const float2 A1 = f2_unpack(v1[0]), B1 = f2_unpack(v1[1]);
      t = f2_pack(lerp(A0.x, B0.x, c2v[0]), lerp(A1.x, B1.x, c2v[1]));
      q = f2_pack(lerp(A0.y, B0.y, c2v[0]), lerp(A1.y, B1.y, c2v[1]));
    };
    const unsigned long long zp = f2_pack(zv[0], zv[1]);
    const unsigned long long z2p = f2_mul(zp, zp);
    const unsigned long long nl0 = f2_pack(-lim[0][0], -lim[0][1]);
    const unsigned long long nl1 = f2_pack(-lim[1][0], -lim[1][1]);
    const unsigned long long nl2 = f2_pack(-lim[2][0], -lim[2][1]);
    const unsigned long long nl3 = f2_pack(-lim[3][0], -lim[3][1]);
    const unsigned long long iw0 = f2_pack(iwv[0][0], iwv[0][1]);
    const unsigned long long iw1 = f2_pack(iwv[1][0], iwv[1][1]);
    const unsigned long long iw2 = f2_pack(iwv[2][0], iwv[2][1]);
    const unsigned long long iw3 = f2_pack(iwv[3][0], iwv[3][1]);
    const unsigned long long two23 = f2_dup(8388608.0f);
    unsigned long long acc = f2_pack(accv[0], accv[1]), cmp = f2_pack(cmpv[0], cmpv[1]);
    const unsigned mybit = 0x10000u << lx;

    for (int s0 = 0; s0 < nsrc; s0 += sc) {
      const int ns = min(sc, nsrc - s0);
      for (int s = 0; s < ns && act[0]; ++s) {
        const float2 sp = srcpos[s0 + s];
        float4 *m = smap4 + s * NT + tid;
        if (!tile_covers(s_tg, sp)) {
          // no table value: NaN fails every member's dip test
          m[0] = m[splane] = m[2 * splane] = m[3 * splane] = make_float4(NAN, NAN, NAN, NAN);
          continue;
        }
        int off;
        float wx, wy;
        surface_weights(s_tg, sp.x, sp.y, plane, off, wx, wy);
        unsigned long long tp, qp;
        lookup(off, wx, wy, tp, qp);
        const float2 ts = f2_unpack(tp), qs = f2_unpack(qp);
        const float dsx = sp.x - x;
        float px1[2], px2[2], py1[2], py2[2], cs[2], azv[2];
#pragma unroll
        for (int p = 0; p < 2; ++p) {
          const float z2 = zv[p] * zv[p];
          const float ds = sqrtf(dsx * dsx + sp.y * sp.y + z2);
          const float rds = __fdividef(1.0f, ds);
          const float ax = dsx * rds, ay = sp.y * rds, az = zv[p] * rds;
          cs[p] = __fdividef(ds * ds * ds, p ? ts.y : ts.x);
          azv[p] = az;
          px1[p] = fmaf(-lim[0][p], az, ax), px2[p] = fmaf(lim[1][p], az, -ax);
          py1[p] = fmaf(-lim[2][p], az, ay), py2[p] = fmaf(lim[3][p], az, -ay);
        }
        m[0] = make_float4(px1[0], px1[1], px2[0], px2[1]);
        m[splane] = make_float4(py1[0], py1[1], py2[0], py2[1]);
        m[2 * splane] = make_float4(ts.x, ts.y, qs.x * inv_dts, qs.y * inv_dts);
        m[3 * splane] = make_float4(cs[0], cs[1], azv[0], azv[1]);
      }
      for (int pc0 = ipart * clen; pc0 < nmem_all; pc0 += nsplit * clen) {
        const int nmem = min(pc0 + clen, nmem_all);
        // keep pass: one bit per member of the chunk
#pragma unroll 4
        for (int k = 0; k < MW / NW; ++k) {
          const int wi = k * NW + warp;
          const int p = pc0 + 32 * wi + lane;
          bool keep = false;
          if (p < nmem) {
            const int4 mi = __ldg(mem + p);
            const int sl = (mi.y & 0xFFFFFF) - s0;
            const int lo = max(mi.z, ixi_lo), hi = min(mi.w, ixi_hi);
            if (sl >= 0 && sl < ns && lo <= hi) {
              const float2 sp = __ldg(srcpos + s0 + sl), gp = __ldg(grppos + __ldg(memgrp + p));
              if (tile_covers(s_tg, sp) && tile_covers(s_tg, gp)) {
                // every active point of columns lo..hi is a point-trace
                const unsigned n = s_col[hi - ixi_lo + 1] - s_col[lo - ixi_lo];
                cnt += n;
                keep = tile_keep(sp, gp, s_box);
                if (!keep) cdrop += n;
              }
            }
          }
          const unsigned bits = __ballot_sync(0xffffffffu, keep);
          if (lane == 0) s_mask[wi] = bits;
        }
        __syncthreads();
        if (warp == 0) {  // exclusive prefix of the words' kept counts
          int run = 0;
          for (int w0 = 0; w0 < MW; w0 += 32) {
            const int w = w0 + lane;
            int c = w < MW ? __popc(s_mask[w]) : 0;
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) {
              const int v = __shfl_up_sync(0xffffffffu, c, off);
              if (lane >= off) c += v;
            }
            if (w < MW) s_wpos[w + 1] = run + c;
            run += __shfl_sync(0xffffffffu, c, 31);
          }
          if (lane == 0) s_wpos[0] = 0;
        }
        __syncthreads();
        // the kept members' records, in member order
#pragma unroll 2
        for (int k = 0; k < MW / NW; ++k) {
          const int wi = k * NW + warp;
          const unsigned bits = s_mask[wi];
          if (!((bits >> lane) & 1u)) continue;
          const int p = pc0 + 32 * wi + lane;
          const int4 mi = __ldg(mem + p);
          const int sl = (mi.y & 0xFFFFFF) - s0, g = __ldg(memgrp + p);
          const unsigned below = bits & ((1u << lane) - 1u);
          // the kept member before this one, in this or an earlier word
          int prev = -1;
          if (below) {
            prev = pc0 + 32 * wi + 31 - __clz(below);
          } else {
            for (int w = wi - 1; w >= 0; --w)
              if (s_mask[w]) {
                prev = pc0 + 32 * w + 31 - __clz(s_mask[w]);
                break;
              }
          }
          const bool fresh = prev < 0 || __ldg(memgrp + prev) != g;
          const int lo = max(mi.z, ixi_lo) - ixi_lo, hi = min(mi.w, ixi_hi) - ixi_lo;
          const unsigned cols = (0xFFFFu >> (15 - hi)) & (0xFFFFu << lo);
          const float2 gp = __ldg(grppos + g);
          int off;
          float wx, wy;
          surface_weights(s_tg, gp.x, gp.y, plane, off, wx, wy);
          // 2^e of the trace's FP16 panel from the record's exponent bits
          float scale = 100.0f;
          if (std::is_same<T, __half>::value)
            scale *= __int_as_float((int)((((unsigned)mi.y >> 24) - 1u) << 23));
          const int at = s_wpos[wi] + __popc(below);
          s_rec[at] = make_int4(mi.x, (int)(cols << 16) | (fresh ? kNewGroup : 0) | sl, off,
                                __float_as_int(scale));
          s_geo[at] = make_float4(gp.x, gp.y, wx, wy);
        }
        if (tid < U) s_rec[s_wpos[MW] + tid] = make_int4(0, kNewGroup, 0, 0);  // ends a block
        __syncthreads();
        const int nkept = s_wpos[MW];
        if (act[0] && nkept > 0) {
          unsigned long long agz = 0, q0 = 0, q1 = 0, q2 = 0, q3 = 0, tg = 0, qg = 0, gfac = 0;
          int4 nx = s_rec[0];
          for (int k = 0; k < nkept;) {
            int4 rec[U];
            rec[0] = nx;
            if (rec[0].y & kNewGroup) {
              // receiver terms, once per receiver position
              const float4 ge = s_geo[k];
              lookup(rec[0].z, ge.z, ge.w, tg, qg);
              const float dgx = ge.x - x;
              const float2 d2 = f2_unpack(f2_add(f2_dup(dgx * dgx + ge.y * ge.y), z2p));
              const unsigned long long rdg = f2_pack(rsqrt_fast(d2.x), rsqrt_fast(d2.y));
              const unsigned long long agx = f2_mul(f2_dup(dgx), rdg);
              const unsigned long long agy = f2_mul(f2_dup(ge.y), rdg);
              agz = f2_mul(zp, rdg);
              // dip-test thresholds of this receiver: q0, q2 with opposite sign
              q0 = f2_fma(nl0, agz, agx);
              q1 = f2_fma(nl1, agz, agx);
              q2 = f2_fma(nl2, agz, agy);
              q3 = f2_fma(nl3, agz, agy);
              gfac = f2_mul(f2_mul(f2_mul(tg, rdg), rdg), rdg);
              qg = f2_mul(qg, f2_dup(inv_dts));
            }
            // up to U kept members of this receiver
            bool take[U];
            take[0] = true;
            ++k;
            nx = s_rec[k];
#pragma unroll
            for (int u = 1; u < U; ++u) {
              rec[u] = nx;
              take[u] = take[u - 1] && !(nx.y & kNewGroup);
              if (take[u]) {
                ++k;
                nx = s_rec[k];
              }
            }
            bool on[U][2], any = false;
            float4 F0[U], F1[U];
            const float2 q0v = f2_unpack(q0), q1v = f2_unpack(q1);
            const float2 q2v = f2_unpack(q2), q3v = f2_unpack(q3);
#pragma unroll
            for (int u = 0; u < U; ++u) {
              const float4 *m = smap4 + (rec[u].y & 0xFF) * NT + tid;
              F0[u] = m[0];
              F1[u] = m[splane];
              const bool inr = take[u] && ((unsigned)rec[u].y & mybit);
              on[u][0] = inr && F0[u].x > -q0v.x && F0[u].z > q1v.x && F1[u].x > -q2v.x &&
                         F1[u].z > q3v.x;
              on[u][1] = inr && F0[u].y > -q0v.y && F0[u].w > q1v.y && F1[u].y > -q2v.y &&
                         F1[u].w > q3v.y;
              any = any || on[u][0] || on[u][1];
            }
            if (!any) continue;
            unsigned long long fwt[U], fwb[U], fac[U];
            const T *pp[U][2];
#pragma unroll
            for (int u = 0; u < U; ++u) {
              const float4 *m = smap4 + (rec[u].y & 0xFF) * NT + tid;
              const float4 F2 = m[2 * splane], F3 = m[3 * splane];
              const unsigned long long t = f2_add(f2_pack(F2.x, F2.y), tg);
              const unsigned long long ft = f2_mul(t, f2_dup(inv_dt1));
              // floor in the low bits (ft < 0, ft past 2^23 and NaN fail the window test)
              const unsigned long long mt = f2_add_rz(ft, two23);
              fwt[u] = f2_sub(ft, f2_sub(mt, two23));
              const float2 fbr = f2_unpack(f2_add(f2_pack(F2.z, F2.w), qg));
              const unsigned long long fb = f2_pack(fminf(fmaxf(fbr.x, 0.0f), fb_max),
                                                    fminf(fmaxf(fbr.y, 0.0f), fb_max));
              const unsigned long long mb = f2_add_rz(fb, two23);
              fwb[u] = f2_sub(fb, f2_sub(mb, two23));
              const float2 mtv = f2_unpack(mt), mbv = f2_unpack(mb);
              const unsigned it0 = __float_as_uint(mtv.x), it1 = __float_as_uint(mtv.y);
              on[u][0] = on[u][0] && it0 - 0x4B000001u < (unsigned)(a.nt - 2);
              on[u][1] = on[u][1] && it1 - 0x4B000001u < (unsigned)(a.nt - 2);
              const T *pt = panels + (uint64_t)(unsigned)rec[u].x * pstride;
              pp[u][0] = pt + (__float_as_uint(mbv.x) * (unsigned)a.nt + it0 - idx0);
              pp[u][1] = pt + (__float_as_uint(mbv.y) * (unsigned)a.nt + it1 - idx0);
              // dip taper and w v (r + 1/r) = w (r^2 + 1) 100 / (r tt)
              const unsigned long long uz = f2_add(f2_pack(F3.z, F3.w), agz);
              const float2 e0 = f2_unpack(f2_mul(f2_add(f2_pack(F0[u].x, F0[u].y), q0), iw0));
              const float2 e1 = f2_unpack(f2_mul(f2_sub(f2_pack(F0[u].z, F0[u].w), q1), iw1));
              const float2 e2 = f2_unpack(f2_mul(f2_add(f2_pack(F1[u].x, F1[u].y), q2), iw2));
              const float2 e3 = f2_unpack(f2_mul(f2_sub(f2_pack(F1[u].z, F1[u].w), q3), iw3));
              const unsigned long long r = f2_mul(f2_pack(F3.x, F3.y), gfac);
              const float2 tv = f2_unpack(t), t2 = f2_unpack(f2_mul(t, t));
              const unsigned long long rtt =
                  f2_mul(r, f2_pack(tv.x > 0.1f ? t2.x : 0.01f, tv.y > 0.1f ? t2.y : 0.01f));
              const float2 den = f2_unpack(f2_mul(uz, rtt));
              const unsigned long long inv = f2_pack(rcp_fast(den.x), rcp_fast(den.y));
              const unsigned long long ruz = f2_mul(rtt, inv);
              const float2 ex =
                  f2_unpack(f2_mul(f2_pack(fminf(e0.x, e1.x), fminf(e0.y, e1.y)), ruz));
              const float2 ey =
                  f2_unpack(f2_mul(f2_pack(fminf(e2.x, e3.x), fminf(e2.y, e3.y)), ruz));
              const unsigned long long wt = f2_mul(f2_pack(fminf(1.0f, ex.x), fminf(1.0f, ex.y)),
                                                   f2_pack(fminf(1.0f, ey.x), fminf(1.0f, ey.y)));
              const float2 fv = f2_unpack(
                  f2_mul(f2_mul(wt, f2_fma(r, r, f2_dup(1.0f))),
                         f2_mul(f2_mul(f2_dup(__int_as_float(rec[u].w)), uz), inv)));
              // a lane that is off adds 0 times an interpolation of zeros: its factor
              // and, since t may be infinite or NaN there, its time weight are 0
              // (0.2 % of the kernel; choosing between the old and the new sum took 6 %)
              fac[u] = f2_pack(on[u][0] ? fv.x : 0.0f, on[u][1] ? fv.y : 0.0f);
              const float2 wv = f2_unpack(fwt[u]);
              fwt[u] = f2_pack(on[u][0] ? wv.x : 0.0f, on[u][1] ? wv.y : 0.0f);
              cimg += on[u][0];
              cimg += on[u][1];
            }
            float sm[U][2][4];
#pragma unroll
            for (int u = 0; u < U; ++u)
#pragma unroll
              for (int p = 0; p < 2; ++p) {
                sm[u][p][0] = sm[u][p][1] = sm[u][p][2] = sm[u][p][3] = 0.0f;
                if (on[u][p]) {
                  const T *q = pp[u][p];
                  sm[u][p][0] = ld_sample<T>(q);
                  sm[u][p][1] = ld_sample<T>(q + 1);
                  sm[u][p][2] = ld_sample<T>(q + a.nt);
                  sm[u][p][3] = ld_sample<T>(q + a.nt + 1);
                }
              }
#pragma unroll
            for (int u = 0; u < U; ++u) {
              const unsigned long long p00 = f2_pack(sm[u][0][0], sm[u][1][0]);
              const unsigned long long p01 = f2_pack(sm[u][0][1], sm[u][1][1]);
              const unsigned long long p10 = f2_pack(sm[u][0][2], sm[u][1][2]);
              const unsigned long long p11 = f2_pack(sm[u][0][3], sm[u][1][3]);
              const unsigned long long v = f2_lerp(f2_lerp(p00, p01, fwt[u]),
                                                   f2_lerp(p10, p11, fwt[u]), fwb[u]);
              if (comp) {  // Kahan-compensated sums (a point that is off adds zero)
                const unsigned long long y = f2_sub(f2_mul(fac[u], v), cmp);
                const unsigned long long tt = f2_add(acc, y);
                cmp = f2_sub(f2_sub(tt, acc), y);
                acc = tt;
              } else {
                acc = f2_fma(fac[u], v, acc);
              }
            }
          }
        }
        __syncthreads();  // s_mask, s_wpos, s_rec and s_geo are rewritten by the next chunk
      }
    }
    const float2 av = f2_unpack(acc), cv = f2_unpack(cmp);
    const size_t o = (size_t)ixb * a.nzi + izi;
    if (nsplit == 1) {
#pragma unroll
      for (int p = 0; p < 2; ++p)
        if (live[p]) {
          img[o + p] = p ? av.y : av.x;
          if (comp) comp[o + p] = p ? cv.y : cv.x;
        }
      continue;
    }
    const size_t nimg = (size_t)a.nxb * a.nzi;
#pragma unroll
    for (int p = 0; p < 2; ++p)
      if (live[p])
        put_part(part + o + p, nimg, ipart, p ? av.y : av.x, p ? cv.y : cv.x, comp);
    if (!last_part(tile_done + tile, nsplit, &s_tile)) continue;
#pragma unroll
    for (int p = 0; p < 2; ++p)
      if (live[p])
        add_parts(img + o + p, comp ? comp + o + p : nullptr, part + o + p, nimg, nsplit);
  }
  if (npt) add_counts(npt, s_cnt, cnt, cdrop, cimg);
}

static int batched_alloc(PhysicsState *s, const qpsdm_static_params &p) {
  const int n = p.max_batch;
  bool ok = true;
  for (GroupSet &g : s->sets) {
    for (int i = 0; i < 2; ++i) {
      ok &= cudaMalloc(&g.d_key[i], sizeof(unsigned long long) * n) == cudaSuccess;
      ok &= cudaMalloc(&g.d_val[i], sizeof(int) * n) == cudaSuccess;
    }
    ok &= cudaMalloc(&g.d_ukey, sizeof(unsigned long long) * n) == cudaSuccess;
    ok &= cudaMalloc(&g.d_count, sizeof(int) * n) == cudaSuccess;
    ok &= cudaMalloc(&g.d_off, sizeof(int) * n) == cudaSuccess;
    ok &= cudaMalloc(&g.d_nruns, sizeof(int)) == cudaSuccess;
    ok &= cudaMalloc(&g.d_srcflag, sizeof(int) * n) == cudaSuccess;
    ok &= cudaMalloc(&g.d_sid, sizeof(int) * n) == cudaSuccess;
    ok &= cudaMalloc(&g.d_srcpos, sizeof(float2) * n) == cudaSuccess;
    ok &= cudaMalloc(&g.d_mem, sizeof(int4) * n) == cudaSuccess;
    ok &= cudaMalloc(&g.d_grppos, sizeof(float2) * n) == cudaSuccess;
    ok &= cudaMalloc(&g.d_memgrp, sizeof(int) * n) == cudaSuccess;
    ok &= cudaMalloc(&g.d_nmem, sizeof(int)) == cudaSuccess;
  }
  if (!ok) return QPSDM_ENOMEM;
  GroupSet &g0 = s->sets[0];
  size_t b1 = 0, b2 = 0, b3 = 0, b4 = 0;
  cub::DeviceRadixSort::SortPairs(nullptr, b1, g0.d_key[0], g0.d_key[1], g0.d_val[0],
                                  g0.d_val[1], n);
  cub::DeviceRunLengthEncode::Encode(nullptr, b2, g0.d_key[1], g0.d_ukey, g0.d_count,
                                     g0.d_nruns, n);
  cub::DeviceScan::ExclusiveSum(nullptr, b3, g0.d_count, g0.d_off, n);
  cub::DeviceScan::InclusiveSum(nullptr, b4, g0.d_srcflag, g0.d_sid, n);
  s->cub_bytes = std::max(std::max(b1, b2), std::max(b3, b4));
  for (GroupSet &g : s->sets)
    if (cudaMalloc(&g.d_cub, s->cub_bytes) != cudaSuccess) return QPSDM_ENOMEM;
  if (cudaStreamCreateWithFlags(&s->aux, cudaStreamNonBlocking) != cudaSuccess ||
      cudaEventCreateWithFlags(&s->ev_fork, cudaEventDisableTiming) != cudaSuccess ||
      cudaEventCreateWithFlags(&s->ev_join, cudaEventDisableTiming) != cudaSuccess)
    return QPSDM_ECUDA;
  select_set(s, 0);
  int dev = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&s->num_sms, cudaDevAttrMultiProcessorCount, dev);
  if (p.tile_z > 0) s->tile_z = p.tile_z;
  if (p.tile_x > 0) s->tile_x = p.tile_x;
  s->forced_variant = p.variant;
  return QPSDM_OK;
}

// One line of the brick as the image kernels see it.
struct LineView {
  const int *ints;
  const float *geom;
  const float *dips;
  float *img;
  float *comp;
  const PhysicsState::LineTab *tab;
  const qpsdm_line_params *l;
};

// Launch variants of the batched kernel: image tile (depth x cdps, one
// thread per point; a warp spans min(TZ, 32) depths), the minimum resident
// blocks per SM the register allocation is held to, the sources per
// shared-memory chunk (more sources per chunk: fewer passes over the receiver
// groups, more shared memory per block) and the members per block U.  The
// autotuner times them all on the first batch and keeps the fastest.  (U = 8
// was slower everywhere tried: the extra registers cost more occupancy than
// the extra loads in flight gain.)
// Variants from 13 on are the fast form (k_image_batched_fast, with
// k_image_batched over the tiles it leaves) with mw words of 32 members per
// chunk.  16 x 16 tiles of 128 threads at 96 registers (five CTAs, 20 warps
// an SM) win wherever images are large: against 64-thread tiles the keep pass
// and the chunk's barriers serve twice the points, against 128 registers the
// fourth warp per scheduler hides more of the panel loads than the spilled
// words cost.
struct BatchedVariant {
  int tz, tx, mb, sc, u, mw;
};
static const BatchedVariant kVariants[] = {
    {32, 8, 2, 8, 4, 0},  {32, 4, 4, 8, 4, 0},  {32, 4, 6, 8, 4, 0},
    {64, 4, 3, 8, 4, 0},  {32, 4, 3, 16, 4, 0}, {8, 16, 4, 8, 4, 0},
    {4, 32, 4, 8, 4, 0},  {16, 8, 4, 8, 4, 0},  {8, 16, 4, 16, 4, 0},
    {16, 8, 3, 16, 4, 0}, {8, 16, 5, 8, 4, 0},  {8, 16, 5, 16, 4, 0},
    {16, 8, 5, 8, 4, 0},  {8, 16, 8, 4, 1, 8},  {8, 16, 8, 4, 2, 8},
    {16, 8, 8, 4, 2, 8},  {32, 4, 8, 4, 2, 8},  {8, 16, 5, 8, 2, 8},
    {16, 8, 5, 8, 2, 8},  {8, 16, 10, 4, 1, 8}, {8, 16, 5, 8, 1, 8},
    {16, 8, 10, 4, 1, 8}, {8, 16, 6, 4, 2, 8},  {8, 16, 8, 2, 2, 8},
    {8, 16, 8, 4, 2, 16}, {16, 16, 5, 4, 1, 8}, {16, 16, 4, 4, 1, 8},
};
constexpr int kNumVariants = sizeof(kVariants) / sizeof(kVariants[0]);
static_assert(kNumVariants <= 32, "tune_ms holds 32 timings");

// Parts of a tile's members for an image of ntiles tiles: 32 queue items per
// SM, of at least 64 members each, as far as the sums have room.  Tiles differ
// in work by an order of magnitude (the middle of the aperture keeps most
// members, its rim few), so one item per tile leaves most SMs waiting for a
// few: a 512 x 400 line of 18,432 traces (800 tiles of 16 x 16) took 6.3 ms
// in one part per tile, the SMs active 60 % of the time, and 3.1 ms in six;
// 16, 48 and 128 items per SM were no faster.  A 128 x 100 line of 1,024
// traces: 1.29 ms unsplit, 0.08 ms split.  An image of more tiles than that
// is not split (1024 x 600: 2,432 tiles, 38.1 ms against 38.3 for eight lines).
static int member_split(const PhysicsState *s, const PhysImageArgs &a, int ntiles, int ntr) {
  const int want = (32 * s->num_sms + ntiles - 1) / ntiles;
  const size_t room = s->part_cap / (s->part_words * (size_t)a.nxb * a.nzi);
  return std::max(1, std::min(std::min(want, ntr / 64), std::min((int)room, kMaxSplit)));
}

// The original kernel over every tile of the image, or (tile_list) over the
// *ntile_list tiles of a list, with one persistent CTA per SM.
template <int TZ, int TX, int MB, int U, typename T>
static int launch_batched_tile(PhysicsState *s, const PhysImageArgs &a, const PhysicsBatch &b,
                               const LineView &v, float *img, float *comp,
                               unsigned long long *npt, int sc, cudaStream_t st,
                               const int *tile_list = nullptr,
                               const int *ntile_list = nullptr) {
  const int ntz = (a.nzi + TZ - 1) / TZ, ntx = (a.nxb + TX - 1) / TX, ntiles = ntz * ntx;
  const size_t smem = sizeof(float2) * kMapN * (size_t)sc * TZ * TX;
  auto kern = k_image_batched<TZ, TX, MB, U, T>;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) !=
      cudaSuccess)
    return QPSDM_ECUDA;
  int per_sm = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, TZ * TX, smem);
  const int nsplit = member_split(s, a, ntiles, b.ntr);
  const int grid =
      tile_list ? std::max(1, s->num_sms)
                : std::max(1, std::min(ntiles * nsplit, std::max(per_sm, 1) * s->num_sms));
  // the queue's counter and, unless the tiles come from the fast form's list
  // (which has cleared them), the finished parts
  cudaMemsetAsync(s->d_tile_ctr, 0,
                  sizeof(int) * (size_t)(!tile_list && nsplit > 1 ? 2 + ntiles : 1), st);
  kern<<<grid, TZ * TX, smem, st>>>(img, comp, a, v.dips, s->d_memgrp, s->d_grppos, s->d_mem,
                                    s->d_nmem, s->d_srcpos, s->d_sid + (b.ntr - 1), v.tab->dt,
                                    v.tab->ttt, v.tab->dq, v.tab->qqq,
                                    v.tab->paired ? v.tab->tq : nullptr, (const T *)s->d_panels,
                                    s->d_tile_ctr, ntz, ntx, sc, npt, tile_list, ntile_list,
                                    nsplit, s->d_part, s->d_tile_ctr + 2);
  return cudaGetLastError() == cudaSuccess ? QPSDM_OK : QPSDM_ECUDA;
}

// Whether every tile of the image is uniform (k_image_batched_fast leaves
// none): one depth cell, one surface grid, and tile columns that do not
// straddle the tables' x-cells.
static bool all_uniform(const PhysImageArgs &a, const PhysicsState::LineTab &t, int tx) {
  return t.one_grid && a.nzg == 1 && a.nxi1 % tx == 0 && (a.ixstart - a.tcdp1) % tx == 0;
}

// The fast form over the image's uniform tiles, then the original kernel
// (same tile shape, MBO blocks per SM) over the tiles it left; with unpaired
// tables the original kernel takes every tile.
template <int TZ, int TX, int MB, int U, int MW, int MBO, typename T>
static int launch_batched_fast(PhysicsState *s, const PhysImageArgs &a, const PhysicsBatch &b,
                               const LineView &v, float *img, float *comp,
                               unsigned long long *npt, int sc, cudaStream_t st) {
  if (!v.tab->paired)
    return launch_batched_tile<TZ, TX, MBO, 4, T>(s, a, b, v, img, comp, npt, sc, st);
  const int ntz = (a.nzi + TZ - 1) / TZ, ntx = (a.nxb + TX - 1) / TX, ntiles = ntz * ntx;
  if ((size_t)ntiles > s->defer_cap) return QPSDM_EINVAL;  // cannot happen: sized per offset
  const size_t smem = sizeof(float4) * 2 * (size_t)sc * TZ * TX;
  auto kern = k_image_batched_fast<TZ, TX, MB, U, MW, T>;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) !=
      cudaSuccess)
    return QPSDM_ECUDA;
  int per_sm = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, TZ * TX / 2, smem);
  const int nsplit = member_split(s, a, ntiles, b.ntr);
  const int grid = std::max(1, std::min(ntiles * nsplit, std::max(per_sm, 1) * s->num_sms));
  // queue counter, deferred-tile count and the split tiles' finished parts
  cudaMemsetAsync(s->d_tile_ctr, 0, sizeof(int) * (size_t)(nsplit > 1 ? 2 + ntiles : 2), st);
  kern<<<grid, TZ * TX / 2, smem, st>>>(
      img, comp, a, v.dips, s->d_memgrp, s->d_grppos, s->d_mem, s->d_nmem, s->d_srcpos,
      s->d_sid + (b.ntr - 1), v.tab->dt, v.tab->dq, v.tab->tq, (const T *)s->d_panels,
      s->d_tile_ctr, ntz, ntx, sc, npt, s->d_defer, s->d_ndefer, nsplit, s->d_part,
      s->d_tile_ctr + 2);
  if (cudaGetLastError() != cudaSuccess) return QPSDM_ECUDA;
  if (all_uniform(a, *v.tab, TX)) return QPSDM_OK;
  return launch_batched_tile<TZ, TX, MBO, 4, T>(s, a, b, v, img, comp, npt, sc, st, s->d_defer,
                                                s->d_ndefer);
}

template <typename T>
static int launch_variant(int vi, PhysicsState *s, const PhysImageArgs &a, const PhysicsBatch &b,
                          const LineView &v, float *img, float *comp, unsigned long long *npt,
                          cudaStream_t st) {
  const int sc = kVariants[vi].sc;
  switch (vi) {
    case 13: return launch_batched_fast<8, 16, 8, 1, 8, 4, T>(s, a, b, v, img, comp, npt, sc, st);
    case 14:
    case 23: return launch_batched_fast<8, 16, 8, 2, 8, 4, T>(s, a, b, v, img, comp, npt, sc, st);
    case 15: return launch_batched_fast<16, 8, 8, 2, 8, 4, T>(s, a, b, v, img, comp, npt, sc, st);
    case 16: return launch_batched_fast<32, 4, 8, 2, 8, 4, T>(s, a, b, v, img, comp, npt, sc, st);
    case 17: return launch_batched_fast<8, 16, 5, 2, 8, 4, T>(s, a, b, v, img, comp, npt, sc, st);
    case 18: return launch_batched_fast<16, 8, 5, 2, 8, 4, T>(s, a, b, v, img, comp, npt, sc, st);
    case 19: return launch_batched_fast<8, 16, 10, 1, 8, 4, T>(s, a, b, v, img, comp, npt, sc, st);
    case 20: return launch_batched_fast<8, 16, 5, 1, 8, 4, T>(s, a, b, v, img, comp, npt, sc, st);
    case 21: return launch_batched_fast<16, 8, 10, 1, 8, 4, T>(s, a, b, v, img, comp, npt, sc, st);
    case 22: return launch_batched_fast<8, 16, 6, 2, 8, 4, T>(s, a, b, v, img, comp, npt, sc, st);
    case 24: return launch_batched_fast<8, 16, 8, 2, 16, 4, T>(s, a, b, v, img, comp, npt, sc, st);
    case 25: return launch_batched_fast<16, 16, 5, 1, 8, 2, T>(s, a, b, v, img, comp, npt, sc, st);
    case 26: return launch_batched_fast<16, 16, 4, 1, 8, 2, T>(s, a, b, v, img, comp, npt, sc, st);
    case 0: return launch_batched_tile<32, 8, 2, 4, T>(s, a, b, v, img, comp, npt, sc, st);
    case 1: return launch_batched_tile<32, 4, 4, 4, T>(s, a, b, v, img, comp, npt, sc, st);
    case 2: return launch_batched_tile<32, 4, 6, 4, T>(s, a, b, v, img, comp, npt, sc, st);
    case 3: return launch_batched_tile<64, 4, 3, 4, T>(s, a, b, v, img, comp, npt, sc, st);
    case 4: return launch_batched_tile<32, 4, 3, 4, T>(s, a, b, v, img, comp, npt, sc, st);
    case 5: return launch_batched_tile<8, 16, 4, 4, T>(s, a, b, v, img, comp, npt, sc, st);
    case 6: return launch_batched_tile<4, 32, 4, 4, T>(s, a, b, v, img, comp, npt, sc, st);
    case 7: return launch_batched_tile<16, 8, 4, 4, T>(s, a, b, v, img, comp, npt, sc, st);
    case 8: return launch_batched_tile<8, 16, 4, 4, T>(s, a, b, v, img, comp, npt, sc, st);
    case 9: return launch_batched_tile<16, 8, 3, 4, T>(s, a, b, v, img, comp, npt, sc, st);
    case 10:
    case 11: return launch_batched_tile<8, 16, 5, 4, T>(s, a, b, v, img, comp, npt, sc, st);
    case 12: return launch_batched_tile<16, 8, 5, 4, T>(s, a, b, v, img, comp, npt, sc, st);
    default: return QPSDM_EINVAL;
  }
}

// Tuning results shared by the engines of a process:
// (device, nzi, nxb, dtype, nbins, paired tables, batch class) -> variant.  The
// last two decide which kernels run and in how many parts a tile's members are:
// what is fastest for a small batch, or for float tables, is not for the others.
static std::mutex g_tune_mu;
static std::map<std::tuple<int, int, int, int, int, int, int>, int> g_tune;

// Picks the variant for this image shape: an explicit tile from the static
// parameters, a cached result, or a timing of every variant on this batch
// into a scratch image (synchronous; happens on the first batch only).
template <typename T>
static int choose_variant(PhysicsState *s, const PhysImageArgs &a, const PhysicsBatch &b,
                          const LineView &v, cudaStream_t st) {
  if (s->variant >= 0) return s->variant;
  if (s->forced_variant > 0 && s->forced_variant <= kNumVariants)
    return s->variant = s->forced_variant - 1;
  if (s->tile_z > 0 && s->tile_x > 0) {
    for (int i = 0; i < kNumVariants; ++i)
      if (kVariants[i].tz == s->tile_z && kVariants[i].tx == s->tile_x) return s->variant = i;
  }
  int dev = 0;
  cudaGetDevice(&dev);
  int parts = 0;  // log2 of the parts of 16 x 16 tiles: six classes
  for (int n = member_split(s, a, (a.nzi + 15) / 16 * ((a.nxb + 15) / 16), b.ntr); n > 1; n /= 2)
    ++parts;
  const auto key = std::make_tuple(dev, a.nzi, a.nxb, s->dtype, s->nbins, (int)v.tab->paired, parts);
  {
    std::lock_guard<std::mutex> lk(g_tune_mu);
    auto it = g_tune.find(key);
    if (it != g_tune.end()) return s->variant = it->second;
  }
  float *scratch = s->d_tune;
  const size_t n = (size_t)a.nxb * a.nzi;
  if (!scratch || s->tune_cap < n) return s->variant = 2;
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  int best = 2;
  float best_ms = 1e30f;
  for (int i = 0; i < kNumVariants; ++i) {
    cudaMemsetAsync(scratch, 0, sizeof(float) * n, st);
    cudaEventRecord(e0, st);
    const int rc = launch_variant<T>(i, s, a, b, v, scratch, nullptr, nullptr, st);
    cudaEventRecord(e1, st);
    if (rc || cudaEventSynchronize(e1) != cudaSuccess) continue;
    float ms = 0.0f;
    cudaEventElapsedTime(&ms, e0, e1);
    s->tune_ms[i] = ms;
    if (ms < best_ms) {
      best_ms = ms;
      best = i;
    }
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  cudaGetLastError();
  std::lock_guard<std::mutex> lk(g_tune_mu);
  g_tune[key] = best;
  return s->variant = best;
}

template <typename T>
static int launch_batched_image(PhysicsState *s, const PhysImageArgs &a, const PhysicsBatch &b,
                                const LineView &v, cudaStream_t st) {
  const int vi = choose_variant<T>(s, a, b, v, st);
  return launch_variant<T>(vi, s, a, b, v, v.img, v.comp, b.d_npt, st);
}

// Grouping of one batch (all on the stream, nothing read back).
static int batched_group(PhysicsState *s, const qpsdm_static_params &p, const LineView &v,
                         const PhysicsBatch &b, cudaStream_t st) {
  const qpsdm_line_params &l = *v.l;
  const int n = b.ntr, blk = 256, grd = (n + blk - 1) / blk;
  cudaMemsetAsync(s->d_nmem, 0, sizeof(int), st);
  k_batch_keys<<<grd, blk, 0, st>>>(b.d_rec, b.rec_bytes, b.big_endian, n, v.ints, v.geom,
                                    s->d_key[0], s->d_val[0], s->d_srcflag, s->d_nmem);
  size_t tb = s->cub_bytes;
  if (cub::DeviceScan::InclusiveSum(s->d_cub, tb, s->d_srcflag, s->d_sid, n, st) != cudaSuccess)
    return QPSDM_ECUDA;
  tb = s->cub_bytes;
  if (cub::DeviceRadixSort::SortPairs(s->d_cub, tb, s->d_key[0], s->d_key[1], s->d_val[0],
                                      s->d_val[1], n, 0, 64, st) != cudaSuccess)
    return QPSDM_ECUDA;
  cudaMemsetAsync(s->d_count, 0, sizeof(int) * n, st);
  tb = s->cub_bytes;
  if (cub::DeviceRunLengthEncode::Encode(s->d_cub, tb, s->d_key[1], s->d_ukey, s->d_count,
                                         s->d_nruns, n, st) != cudaSuccess)
    return QPSDM_ECUDA;
  tb = s->cub_bytes;
  if (cub::DeviceScan::ExclusiveSum(s->d_cub, tb, s->d_count, s->d_off, n, st) != cudaSuccess)
    return QPSDM_ECUDA;
  k_batch_groups<<<grd, blk, 0, st>>>(s->d_ukey, s->d_nruns, s->d_grppos, n);
  k_batch_memgrp<<<grd, blk, 0, st>>>(s->d_off, s->d_nruns, s->d_memgrp, n);
  k_batch_members<<<grd, blk, 0, st>>>(b.d_rec, b.rec_bytes, b.big_endian, n, s->d_val[1],
                                       v.ints, s->d_sid, s->d_srcflag, p.scaled, l.fxi, l.cyi,
                                       s->dtype == QPSDM_PANEL_FP16 ? s->d_pscale : nullptr,
                                       s->d_mem, s->d_srcpos);
  return cudaGetLastError() == cudaSuccess ? QPSDM_OK : QPSDM_ECUDA;
}

// Any line of the brick accepted the trace: its panels are needed.
__global__ void k_any_line(const int *__restrict__ ints, size_t ints_ls, int nlines, int ntr,
                           unsigned long long mask, int *__restrict__ any) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= ntr) return;
  int a = 0;
  for (int il = 0; il < nlines; ++il)
    if (il >= 64 || ((mask >> il) & 1ull))
      a |= ints[il * ints_ls + (size_t)i * kGateInts] == kAccepted;
  any[i] = a ? kAccepted : 0;
}

template <typename T>
static int launch_panels(PhysicsState *s, const FftPlan &pi, const int *status, int sstride,
                         int ntr, int nk, const float *pscale, cudaStream_t st) {
  auto kern = pi.spad ? k_phys_panels<true, T> : k_phys_panels<false, T>;
  const size_t sm = 2 * sizeof(float4) * (size_t)pi.swords + sizeof(float2) * (size_t)s->kmax;
  int rc = fft_set_smem_attr((const void *)kern, sm);
  if (rc) return rc;
  int dev = 0, nsm = 0, per_sm = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, pi.sthreads, sm);
  // as many CTAs as fit; a trace is split into groups of bin pairs until there
  // are eight items per CTA (a group reloads the trace's band, 7 KB)
  const int slots = std::max(per_sm, 1) * std::max(nsm, 1), npairs = (s->nbins + 1) / 2;
  int ngroups = 1;
  while (ngroups < npairs && (int64_t)ntr * ngroups < 8ll * slots) ngroups *= 2;
  ngroups = std::min(ngroups, npairs);
  const int grid = (int)std::max<int64_t>(1, std::min<int64_t>((int64_t)ntr * ngroups, slots));
  kern<<<grid, pi.sthreads, sm, st>>>(status, sstride, ntr, s->d_spec, nk, s->kmax, s->d_filter, pi,
                              s->nbins, ngroups, (T *)s->d_panels, pscale);
  return QPSDM_OK;
}

// Forward spectra and t*-binned panels of the traces whose status is kAccepted.
static int run_panels(PhysicsState *s, const qpsdm_static_params &p, const PhysicsBatch &b,
                      const int *status, int sstride, cudaStream_t st, std::string *err) {
  FftPlan pf, pi;
  int rc = fft_plan(p.nfft, &pf, err);
  if (rc) return rc;
  rc = fft_plan(p.nffti, &pi, err);
  if (rc) return rc;
  const int ntr = b.ntr;
  const bool fp16 = s->dtype == QPSDM_PANEL_FP16;
  const size_t sm = 2 * sizeof(float4) * (size_t)pf.swords;
  auto fwd = pf.spad ? k_phys_fwd<true> : k_phys_fwd<false>;
  if ((rc = fft_set_smem_attr((const void *)fwd, sm))) return rc;
  fwd<<<(ntr + 1) / 2, pf.sthreads, sm, st>>>(b.d_rec, b.rec_bytes, b.big_endian, status, sstride,
                                              ntr, p.ntl, p.dt, b.d_taper200, pf, s->d_spec,
                                              s->d_fmax, fp16 ? s->d_pscale : nullptr);
  const int nk = p.nfft / 2 + 1;
  if (s->dtype == QPSDM_PANEL_FP32)
    rc = launch_panels<float>(s, pi, status, sstride, ntr, nk, nullptr, st);
  else if (s->dtype == QPSDM_PANEL_BF16)
    rc = launch_panels<__nv_bfloat16>(s, pi, status, sstride, ntr, nk, nullptr, st);
  else
    rc = launch_panels<__half>(s, pi, status, sstride, ntr, nk, s->d_pscale, st);
  return rc ? rc : cudaGetLastError() == cudaSuccess ? QPSDM_OK : QPSDM_ECUDA;
}

static PhysImageArgs image_args(const PhysicsState *s, const qpsdm_static_params &p,
                                const qpsdm_line_params &l, const qpsdm_offset_params &o,
                                size_t nxz) {
  PhysImageArgs a{};
  a.nzi = p.nzi;
  a.nxb = o.ixend - o.ixstart;
  a.ixstart = o.ixstart;
  a.nt = p.nffti;
  a.nbins = s->nbins;
  a.dt1 = p.dt1;
  a.dxi = p.dxi;
  a.dzi = p.dzi;
  a.taperzone = p.taperzone;
  a.dtstar = s->dtstar;
  a.dzii = p.dzii;
  a.tcdp1 = l.ttt_cdp1 - p.fci;
  a.tcdp2 = l.ttt_cdp2 - p.fci;
  a.nxg = l.nxg;
  a.nzg = l.nzg;
  a.nxi1 = l.nxi1;
  a.nzi1 = l.nzi1;
  a.nxz = nxz;
  a.xfast = s->form == QPSDM_FORM_BATCHED;
  return a;
}

template <int SPLIT, typename T>
static void launch_plain_split(const PhysImageArgs &a, const PhysicsBatch &b, const LineView &v,
                               const T *panels, const float *pscale, cudaStream_t st) {
  dim3 grid((a.nzi + 31) / 32, (a.nxb + 8 / SPLIT - 1) / (8 / SPLIT));
  k_image_plain<SPLIT, T><<<grid, 256, 0, st>>>(v.img, v.comp, a, v.dips, v.ints, v.geom, b.ntr,
                                                v.tab->dt, v.tab->ttt, v.tab->dq, v.tab->qqq,
                                                v.tab->paired ? v.tab->tq : nullptr, panels,
                                                pscale, b.d_npt);
}

template <typename T>
static void launch_plain(const PhysImageArgs &a, const PhysicsBatch &b, const LineView &v,
                         const T *panels, const float *pscale, cudaStream_t st) {
  ordered_by_split(a.nzi, a.nxb, 16, [&](auto split) {
    launch_plain_split<decltype(split)::value, T>(a, b, v, panels, pscale, st);
  });
}

int physics_process(PhysicsState *s, const qpsdm_static_params &p,
                    const qpsdm_line_params *lines, const qpsdm_offset_params &o,
                    const PhysicsBatch &b, cudaStream_t st, std::string *err) {
  if (s->ntabs < b.nlines) {
    if (err) *err = "physics mode: set_line without tables";
    return QPSDM_ESTATE;
  }
  const size_t nimg = (size_t)(o.ixend - o.ixstart) * p.nzi;
  auto view = [&](int il) {
    LineView v;
    v.ints = b.d_ints + il * b.ints_ls;
    v.geom = b.d_geom + il * b.geom_ls;
    v.dips = b.d_dips + (size_t)il * 4 * b.nxz;
    v.img = b.d_img + il * b.img_ls;
    v.comp = p.kahan ? s->d_comp + il * nimg : nullptr;
    v.tab = &s->tabs[il];
    v.l = &lines[il];
    return v;
  };
  int rc = QPSDM_OK;
  if (s->form == QPSDM_FORM_PLAIN) {
    // (the reference preprocesses its accepted traces again for each line)
    int active = 0, only = 0;
    for (int il = 0; il < b.nlines; ++il)
      if (batch_line_on(b, il)) {
        ++active;
        only = il;
      }
    if (active == 0) return rc;
    b.prof->begin(QPSDM_K_PRE, st);
    if (active > 1)
      k_any_line<<<(b.ntr + 255) / 256, 256, 0, st>>>(b.d_ints, b.ints_ls, b.nlines, b.ntr,
                                                      b.line_mask, s->d_any);
    rc = active > 1 ? run_panels(s, p, b, s->d_any, 1, st, err)
                    : run_panels(s, p, b, view(only).ints, kGateInts, st, err);
    b.prof->end(st);
    for (int il = 0; il < b.nlines && !rc; ++il) {
      if (!batch_line_on(b, il)) continue;
      const LineView v = view(il);
      const PhysImageArgs a = image_args(s, p, lines[il], o, b.nxz);
      b.prof->begin(QPSDM_K_IMAGE, st);
      if (s->dtype == QPSDM_PANEL_FP32)
        launch_plain<float>(a, b, v, (const float *)s->d_panels, s->d_pscale, st);
      else if (s->dtype == QPSDM_PANEL_BF16)
        launch_plain<__nv_bfloat16>(a, b, v, (const __nv_bfloat16 *)s->d_panels, s->d_pscale,
                                    st);
      else
        launch_plain<__half>(a, b, v, (const __half *)s->d_panels, s->d_pscale, st);
      b.prof->end(st);
      if (cudaGetLastError() != cudaSuccess) rc = QPSDM_ECUDA;
    }
    if (rc && err && err->empty()) *err = "physics launch failed";
    return rc;
  }
  // batched: panels once for every trace any line accepted, shared by the brick
  b.prof->begin(QPSDM_K_PRE, st);
  k_any_line<<<(b.ntr + 255) / 256, 256, 0, st>>>(b.d_ints, b.ints_ls, b.nlines, b.ntr,
                                                  b.line_mask, s->d_any);
  rc = run_panels(s, p, b, s->d_any, 1, st, err);
  b.prof->end(st);
  if (rc) return rc;
  // Lines alternate between the engine's stream (grouping set 0) and the
  // second stream (set 1), which starts after the panels; the engine's stream
  // waits for the second one before returning, so the next batch (which
  // rewrites the panels) and any read of the image come after every line.
  int nactive = 0;
  for (int il = 0; il < b.nlines; ++il) nactive += batch_line_on(b, il);
  const bool forked = nactive > 1;
  if (forked && (cudaEventRecord(s->ev_fork, st) != cudaSuccess ||
                 cudaStreamWaitEvent(s->aux, s->ev_fork, 0) != cudaSuccess))
    return QPSDM_ECUDA;
  int nrun = 0;
  for (int il = 0; il < b.nlines && !rc; ++il) {
    if (!batch_line_on(b, il)) continue;
    const int set = nrun++ & 1;
    cudaStream_t ss = set ? s->aux : st;
    select_set(s, set);
    const LineView v = view(il);
    b.prof->begin(QPSDM_K_OTHER, ss);
    rc = batched_group(s, p, v, b, ss);
    b.prof->end(ss);
    if (rc) {
      if (err) *err = "batched grouping failed";
      break;
    }
    const PhysImageArgs a = image_args(s, p, lines[il], o, b.nxz);
    b.prof->begin(QPSDM_K_IMAGE, ss);
    if (s->dtype == QPSDM_PANEL_FP32)
      rc = launch_batched_image<float>(s, a, b, v, ss);
    else if (s->dtype == QPSDM_PANEL_BF16)
      rc = launch_batched_image<__nv_bfloat16>(s, a, b, v, ss);
    else
      rc = launch_batched_image<__half>(s, a, b, v, ss);
    b.prof->end(ss);
    if (rc && err) *err = "batched image launch failed";
  }
  if (forked && (cudaEventRecord(s->ev_join, s->aux) != cudaSuccess ||
                 cudaStreamWaitEvent(st, s->ev_join, 0) != cudaSuccess) && !rc)
    rc = QPSDM_ECUDA;
  select_set(s, 0);
  return rc;
}

int physics_tuning(const PhysicsState *s, int *variant, int *tz, int *tx, int *mb,
                   float *times, int ntimes) {
  if (!s) return QPSDM_ESTATE;
  const int v = s->variant;
  if (variant) *variant = v;
  if (tz) *tz = v >= 0 ? kVariants[v].tz : 0;
  if (tx) *tx = v >= 0 ? kVariants[v].tx : 0;
  if (mb) *mb = v >= 0 ? kVariants[v].mb : 0;
  for (int i = 0; times && i < ntimes && i < kNumVariants; ++i) times[i] = s->tune_ms[i];
  return kNumVariants;
}

void physics_panels(const PhysicsState *s, void **d_panels, float **d_pscale) {
  *d_panels = s->d_panels;
  *d_pscale = s->d_pscale;
}

int physics_finalize_image(PhysicsState *s, float *d_img, size_t n, cudaStream_t st,
                           std::string *err) {
  (void)s;
  (void)d_img;
  (void)n;
  (void)st;
  (void)err;
  return QPSDM_OK;
}

}  // namespace qpsdm

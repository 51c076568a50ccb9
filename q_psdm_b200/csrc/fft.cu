// fft.cu -- FFT plans (twiddle tables per device and length) and the
// standalone batched real transforms of the C ABI.
#include <algorithm>
#include <cmath>
#include <map>
#include <mutex>
#include <utility>

#include "fft.cuh"
#include "internal.h"
#include "qpsdm_engine.h"

namespace qpsdm {

// The longest half-length: two buffers of a Stockham length in one CTA.
constexpr int kFftMaxHalf = 6399;

static std::mutex g_plan_mu;
static std::map<std::pair<int, int>, FftPlan> g_plans;

// Stockham radices of m: powers of two as 4s (and one 2), nines as 3s, then
// 5, 7, 11, 13; a 4 and the 2 after it, and two 3s, make one group.  A length past
// kFftMaxHalf, which may have more groups than a plan holds, gets none: its
// callers refuse it.
static bool factor_radices(int m, FftPlan &p) {
  int rad[32], n = 0, r = m;
  while (r % 4 == 0) { rad[n++] = 4; r /= 4; }
  if (r % 2 == 0) { rad[n++] = 2; r /= 2; }
  const int odd[5] = {3, 5, 7, 11, 13};
  for (int q : odd)
    while (r % q == 0) { rad[n++] = q; r /= q; }
  if (r != 1) return false;
  p.nstock = 0;
  if (m > kFftMaxHalf) return true;
  for (int i = 0; i < n; ++i) {
    const bool two = i + 1 < n && ((rad[i] == 4 && rad[i + 1] == 2) ||
                                   (rad[i] == 3 && rad[i + 1] == 3));
    p.stock[p.nstock++] = rad[i] + 16 * (two ? rad[i + 1] : 1);
    i += two;
  }
  p.spad = m % 2 == 0 && m <= 5000;
  p.swords = p.spad ? m + m / 8 + 1 : m;
  // the CTA size with the least time per transform of an SM: rounds of
  // butterflies (one of q points weighing about q (q + 12)) over the CTAs that
  // shared memory (two buffers and the band) and 96 registers a thread allow
  const int room = 227 * 1024 / (32 * p.swords + 4 * m + 1024);
  double best = 1e30;
  p.sthreads = 256;
  for (int t = 64; t <= kFftMaxThreads; t += 32) {
    double w = 0.0;
    for (int i = 0; i < p.nstock; ++i) {
      const int q = (p.stock[i] & 15) * (p.stock[i] >> 4);
      w += (double)((m / q + t - 1) / t) * q * (q + 12);
    }
    w /= std::max(1, std::min(room, 65536 / (96 * t)));
    if (w < best * 0.999) {
      best = w;
      p.sthreads = t;
    }
  }
  return true;
}

// The passes of a complex length m.  False: a factor outside
// {2, 3, 5, 7, 11, 13}.
static bool fft_factor(int m, FftPlan &p) {
  p.n = 2 * m;
  p.m = m;
  if (!factor_radices(m, p)) return false;
  if (m > kFftMaxHalf) return true;
  int r = m, np = 0;
  auto take = [&](int q, int prime) {
    if (r % q == 0 && r / q % prime != 0) {
      p.radix[np++] = q;
      r /= q;
    }
  };
  take(13, 13);
  take(11, 11);
  take(9, 3);
  take(3, 3);
  take(7, 7);
  take(5, 5);
  for (int e = 16; e >= 2; e /= 2) take(e, 2);
  if (r != 1) {
    p.mode = kFftStockham;
    p.spad = 0;
    p.swords = m;
    p.words = 2 * m;
    p.threads = p.sthreads;
    return true;
  }
  p.npass = np;
  p.mode = m & 1 ? kFftOdd : kFftEven;
  p.words = m & 1 ? m : m + m / 8 + 1;
  for (int i = 0; i < np; ++i) {
    const int q = p.radix[i], M = m / q;
    int inv = 1;
    while (M % q * inv % q != 1) ++inv;
    p.step[i] = (int)((int64_t)inv * M % m);
  }
  // 20 warps per SM (96 registers a thread) over the CTAs shared memory has
  // room for; a CTA of a short length no wider than its widest pass
  const int ctas = std::max(1, std::min(10, (int)(227 * 1024 / (fft_smem_bytes(p) + 1024))));
  p.threads = std::max(64, std::min(kFftMaxThreads, 640 / ctas / 32 * 32));
  return true;
}

int fft_plan(int n, FftPlan *out, std::string *err) {
  if (n < 2 || (n & 1)) {
    if (err) *err = "FFT length must be even and >= 2";
    return QPSDM_EINVAL;
  }
  int dev = 0;
  cudaGetDevice(&dev);
  std::lock_guard<std::mutex> lk(g_plan_mu);
  auto key = std::make_pair(dev, n);
  auto it = g_plans.find(key);
  if (it != g_plans.end()) {
    *out = it->second;
    return QPSDM_OK;
  }
  FftPlan p{};
  if (!fft_factor(n / 2, p)) {
    if (err) *err = "FFT length " + std::to_string(n) + " has a factor outside {2,3,5,7,11,13}";
    return QPSDM_EINVAL;
  }
  if (p.m > kFftMaxHalf) {
    if (err) *err = "FFT length too large for one CTA";
    return QPSDM_EINVAL;
  }
  std::vector<float2> h((size_t)p.m + (size_t)p.m + 1);
  for (int e = 0; e < p.m; ++e) {
    double a = -2.0 * M_PI * (double)e / (double)p.m;
    h[e] = make_float2((float)std::cos(a), (float)std::sin(a));
  }
  for (int k = 0; k <= p.m; ++k) {
    double a = -2.0 * M_PI * (double)k / (double)n;
    h[p.m + k] = make_float2((float)std::cos(a), (float)std::sin(a));
  }
  float2 *d = nullptr;
  if (cudaMalloc(&d, sizeof(float2) * h.size()) != cudaSuccess) {
    if (err) *err = "cudaMalloc of FFT twiddles failed";
    return QPSDM_ENOMEM;
  }
  cudaMemcpy(d, h.data(), sizeof(float2) * h.size(), cudaMemcpyHostToDevice);
  p.tw_m = d;
  p.tw_n = d + p.m;
  g_plans[key] = p;
  *out = p;
  return QPSDM_OK;
}

// Two transforms per CTA; the last CTA of an odd batch computes its one twice
// and stores it once.  Real rows may be aligned to 4 bytes only.
__device__ __forceinline__ float2 ld_two(const float *x, int j, bool wide) {
  return wide ? reinterpret_cast<const float2 *>(x)[j] : make_float2(x[2 * j], x[2 * j + 1]);
}
__device__ __forceinline__ void st_two(float *y, int j, bool wide, float a, float b) {
  if (wide) {
    reinterpret_cast<float2 *>(y)[j] = make_float2(a, b);
  } else {
    y[2 * j] = a;
    y[2 * j + 1] = b;
  }
}

template <int MODE>
__global__ void __launch_bounds__(kFftMaxThreads, 2)
    k_rfft_batch(const float *__restrict__ in, float2 *__restrict__ out, int batch,
                 const __grid_constant__ FftPlan p) {
  extern __shared__ float4 pbuf[];
  const int ia = 2 * blockIdx.x, ib = min(ia + 1, batch - 1);
  const float *xa = in + (size_t)ia * p.n, *xb = in + (size_t)ib * p.n;
  const bool wide = reinterpret_cast<uintptr_t>(in) % 8 == 0;
  for (int j = threadIdx.x; j < p.m; j += blockDim.x) {
    const float2 a = ld_two(xa, j, wide), b = ld_two(xb, j, wide);
    pbuf[pfa_slot<MODE>(j)] = make_float4(a.x, b.x, a.y, b.y);
  }
  __syncthreads();
  const float4 *Z = fft_passes<MODE>(pbuf, p);
  float2 *ya = out + (size_t)ia * (p.m + 1), *yb = out + (size_t)ib * (p.m + 1);
  for (int k = threadIdx.x; 2 * k <= p.m; k += blockDim.x) {
    const int k2 = p.m - k;
    C2 u, v;
    pfa_rfft_bins(pfa_ld(Z, pfa_slot<MODE>(k)), pfa_ld(Z, pfa_slot<MODE>(k ? k2 : 0)),
                  __ldg(p.tw_n + k), u, v);
    const float2 ur = f2_unpack(u.re), ui = f2_unpack(u.im);
    const float2 vr = f2_unpack(v.re), vi = f2_unpack(v.im);
    ya[k] = make_float2(ur.x, ui.x);
    ya[k2] = make_float2(vr.x, vi.x);
    if (ib != ia) {
      yb[k] = make_float2(ur.y, ui.y);
      yb[k2] = make_float2(vr.y, vi.y);
    }
  }
}

template <int MODE>
__global__ void __launch_bounds__(kFftMaxThreads, 2)
    k_irfft_batch(const float2 *__restrict__ in, float *__restrict__ out, int batch,
                  const __grid_constant__ FftPlan p) {
  extern __shared__ float4 pbuf[];
  const int ia = 2 * blockIdx.x, ib = min(ia + 1, batch - 1);
  const float2 *xa = in + (size_t)ia * (p.m + 1), *xb = in + (size_t)ib * (p.m + 1);
  // real and imaginary parts exchanged: the inverse transform by the forward
  // passes
  for (int k = threadIdx.x; 2 * k <= p.m; k += blockDim.x) {
    const int k2 = p.m - k;
    const float2 a0 = xa[k], b0 = xb[k], a1 = xa[k2], b1 = xb[k2];
    C2 u, v;
    pfa_irfft_pre(C2{f2_pack(a0.x, b0.x), f2_pack(a0.y, b0.y)},
                  C2{f2_pack(a1.x, b1.x), f2_pack(a1.y, b1.y)}, __ldg(p.tw_n + k), u, v);
    pfa_st(pbuf, pfa_slot<MODE>(k), C2{u.im, u.re});
    if (k > 0 && k < k2) pfa_st(pbuf, pfa_slot<MODE>(k2), C2{v.im, v.re});
  }
  __syncthreads();
  const float4 *Z = fft_passes<MODE>(pbuf, p);
  float *ya = out + (size_t)ia * p.n, *yb = out + (size_t)ib * p.n;
  const bool wide = reinterpret_cast<uintptr_t>(out) % 8 == 0;
  for (int j = threadIdx.x; j < p.m; j += blockDim.x) {
    const float4 z = Z[pfa_slot<MODE>(j)];  // (im a, im b, re a, re b)
    st_two(ya, j, wide, 2.0f * z.z, 2.0f * z.x);
    if (ib != ia) st_two(yb, j, wide, 2.0f * z.w, 2.0f * z.y);
  }
}

int fft_set_smem_attr(const void *kernel, size_t bytes) {
  if (bytes > 48 * 1024)
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)bytes) == cudaSuccess
               ? QPSDM_OK
               : QPSDM_ECUDA;
  return QPSDM_OK;
}

static int launch_r2c(const FftPlan &p, const float *d_in, int batch, float *d_out,
                      cudaStream_t st) {
  return fft_by_mode(p, [&](auto mode) {
    auto k = k_rfft_batch<decltype(mode)::value>;
    const size_t sm = fft_smem_bytes(p);
    const int rc = fft_set_smem_attr((const void *)k, sm);
    if (rc) return rc;
    k<<<(batch + 1) / 2, p.threads, sm, st>>>(d_in, (float2 *)d_out, batch, p);
    return cudaGetLastError() == cudaSuccess ? (int)QPSDM_OK : (int)QPSDM_ECUDA;
  });
}

static int launch_c2r(const FftPlan &p, const float *d_in, int batch, float *d_out,
                      cudaStream_t st) {
  return fft_by_mode(p, [&](auto mode) {
    auto k = k_irfft_batch<decltype(mode)::value>;
    const size_t sm = fft_smem_bytes(p);
    const int rc = fft_set_smem_attr((const void *)k, sm);
    if (rc) return rc;
    k<<<(batch + 1) / 2, p.threads, sm, st>>>((const float2 *)d_in, d_out, batch, p);
    return cudaGetLastError() == cudaSuccess ? (int)QPSDM_OK : (int)QPSDM_ECUDA;
  });
}

}  // namespace qpsdm

using namespace qpsdm;

extern "C" int qpsdm_fft_r2c(const float *d_in, int n, int batch, float *d_out,
                             void *stream) {
  if (!d_in || !d_out || batch < 0) return QPSDM_EINVAL;
  if (batch == 0) return QPSDM_OK;
  FftPlan p;
  int rc = fft_plan(n, &p, nullptr);
  if (rc) return rc;
  return launch_r2c(p, d_in, batch, d_out, (cudaStream_t)stream);
}

extern "C" int qpsdm_fft_c2r(const float *d_in, int n, int batch, float *d_out,
                             void *stream) {
  if (!d_in || !d_out || batch < 0) return QPSDM_EINVAL;
  if (batch == 0) return QPSDM_OK;
  FftPlan p;
  int rc = fft_plan(n, &p, nullptr);
  if (rc) return rc;
  return launch_c2r(p, d_in, batch, d_out, (cudaStream_t)stream);
}

// ---------------------------------------------------------------------------
// Allocation-free batched real FFT.
//
// Some callers of this library must not allocate device memory: a host
// framework that owns every byte of HBM through its own pool and forbids
// cudaMalloc behind its back, or a latency-critical caller that cannot take
// the implicit device synchronisation a cudaMalloc may cause.  qpsdm_fft_r2c
// allocates its twiddle tables on the first use of each length; this variant
// keeps them in one fixed file-scope device array instead, which every GPU
// that loads the library holds until the process exits.
//
// The array is shared by every call on a device and keeps the last call's
// twiddles; each call first rewrites the part it uses with a small kernel on
// its own stream (cos and sin of the angles in double precision, rounded once
// to float), so nothing needs clearing and no host buffer is involved.  Calls
// that overlap on the GPU (concurrent streams) race on the array and must be
// serialised by the caller.  The first call on a device looks up the array's
// device address (cudaGetSymbolAddress); make that first call before any
// stream capture.
// ---------------------------------------------------------------------------
namespace qpsdm {

constexpr int kNoAllocMaxDevices = 64;
// m twiddles + (m + 1) split twiddles, m = n / 2 <= QPSDM_FFT_NOALLOC_MAX_N / 2
static __device__ __align__(256) float2 g_noalloc_twiddles[QPSDM_FFT_NOALLOC_MAX_N + 1];
static std::mutex g_noalloc_mu;
static float2 *g_noalloc_dev_ptr[kNoAllocMaxDevices];

// Device address of g_noalloc_twiddles on the current device; set up once per
// device with that device current.  In host code the array's name is only a
// host-side stand-in, never a usable device address.
static int noalloc_twiddle_ptr(float2 **out) {
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kNoAllocMaxDevices)
    return QPSDM_ECUDA;
  std::lock_guard<std::mutex> lk(g_noalloc_mu);
  if (!g_noalloc_dev_ptr[dev]) {
    void *ptr = nullptr;
    if (cudaGetSymbolAddress(&ptr, g_noalloc_twiddles) != cudaSuccess || !ptr)
      return QPSDM_ECUDA;
    g_noalloc_dev_ptr[dev] = (float2 *)ptr;
  }
  *out = g_noalloc_dev_ptr[dev];
  return QPSDM_OK;
}

// Twiddles of length n = 2m into tw: exp(-2 pi i e / m) for e < m, then
// exp(-2 pi i k / n) for k <= m (the layout of FftPlan's tw_m, tw_n).
__global__ void k_noalloc_twiddles(float2 *__restrict__ tw, int m) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= 2 * m + 1) return;
  const double turns = i < m ? -2.0 * (double)i / (double)m : -(double)(i - m) / (double)m;
  double sn, cs;
  sincospi(turns, &sn, &cs);
  tw[i] = make_float2((float)cs, (float)sn);
}

}  // namespace qpsdm

extern "C" int qpsdm_fft_r2c_noalloc(const float *d_in, int n, int batch,
                                     float *d_out, void *stream) {
  if (!d_in || !d_out || batch < 0) return QPSDM_EINVAL;
  if (n > QPSDM_FFT_NOALLOC_MAX_N) return QPSDM_ESIZE;
  if (n < 2 || (n & 1)) return QPSDM_EINVAL;
  if (batch == 0) return QPSDM_OK;
  FftPlan p{};
  if (!fft_factor(n / 2, p) || p.m > kFftMaxHalf) return QPSDM_EINVAL;
  float2 *tw = nullptr;
  int rc = noalloc_twiddle_ptr(&tw);
  if (rc) return rc;
  // this length's twiddles into the shared array, on the caller's stream
  const int ntw = 2 * p.m + 1;
  k_noalloc_twiddles<<<(ntw + 255) / 256, 256, 0, (cudaStream_t)stream>>>(tw, p.m);
  p.tw_m = tw;
  p.tw_n = tw + p.m;
  return launch_r2c(p, d_in, batch, d_out, (cudaStream_t)stream);
}

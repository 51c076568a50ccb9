// fft.cuh -- FFT of two signals at once, in shared memory (sm_100a).
//
// Replaces the reference's host PFA FFT (pfarc/pfacr, src/fft.cc:1768-1910,
// behind the fftw-style shim src/fft.cc:3721-3773).  Real transforms of length
// n use one complex transform of length m = n/2 plus a split step.
//
// Every npfar() length has a half-length m whose factors 2^a, 3^b, 5, 7, 11,
// 13 (a <= 4, b <= 2) are coprime, so the complex transform of length m needs
// no twiddle factors between its passes: the self-sorting in-place prime
// factor algorithm (Temperton, "Implementation of a self-sorting in-place
// prime factor FFT algorithm", J. Comput. Phys. 58, 1985).  A pass of factor
// P transforms each of the m / P sets of points {P u + i m/P mod m} by a
// P-point DFT with constant roots; reading the set in steps of S = r m/P mod m
// (r the inverse of m/P mod P) takes the rotation of the roots out, and every
// output goes back to the set it came from, in natural order in the end.
//
// Two signals share every instruction: a point is (re a, re b, im a, im b),
// one 16-byte word, and the arithmetic runs on f32x2 pairs.
//
// A length with repeated factors (of 2, 3, 5, 7, 11, 13) takes Stockham
// autosort passes (Govindaraju et al., "High performance discrete Fourier
// transforms on graphics processors", SC 2008) over two buffers, with
// twiddles from a table made on the host in double precision.
//
// Measured (c2r, n = 6006, 16,384 transforms): 914 us with one signal per CTA
// in Stockham passes, their roots and twiddles in shared memory; 253 us by the
// prime-factor passes on two signals.
#pragma once

#include <type_traits>

#include "common.cuh"
#include "f32x2.cuh"

namespace qpsdm {

constexpr int kFftMaxPass = 12;
constexpr int kFftMaxThreads = 320;

// How a length is transformed.  A prime-factor pass of an even factor touches
// every P-th word; one word of padding after each 8 spreads those over the
// banks.  Odd lengths have odd factors only.
enum FftMode { kFftOdd = 0, kFftEven = 1, kFftStockham = 2 };

struct FftPlan {
  int n, m;  // real length 2 m, complex length m
  int mode;  // FftMode
  int npass;               // prime-factor passes
  int radix[kFftMaxPass];
  int step[kFftMaxPass];   // S of each
  int nstock;              // Stockham passes: groups of one or two radices,
  int stock[kFftMaxPass];  // PA + 16 PB (PB = 1: one radix)
  int threads;             // CTA size
  int words;               // shared-memory words of the transform
  // the same of the Stockham passes: words of one buffer, padded or not
  int sthreads, swords, spad;
  const float2 *tw_m;     // [m]    exp(-2 pi i e / m)
  const float2 *tw_n;     // [m+1]  exp(-2 pi i k / n)
};
inline size_t fft_smem_bytes(const FftPlan &p) { return 16 * (size_t)p.words; }

// Calls f with the plan's mode as a compile-time constant.
template <typename F>
auto fft_by_mode(const FftPlan &p, F f) {
  switch (p.mode) {
    case kFftOdd: return f(std::integral_constant<int, kFftOdd>());
    case kFftEven: return f(std::integral_constant<int, kFftEven>());
    default: return f(std::integral_constant<int, kFftStockham>());
  }
}

template <int MODE>
__device__ __forceinline__ unsigned pfa_slot(unsigned a) {
  return MODE == kFftEven ? a + (a >> 3) : a;
}
// a mod m for a < 2 m
__device__ __forceinline__ unsigned pfa_wrap(unsigned a, unsigned m) { return min(a, a - m); }

struct C2 {  // one point of two signals
  f2 re, im;
};
__device__ __forceinline__ C2 operator+(C2 a, C2 b) {
  return C2{f2_add(a.re, b.re), f2_add(a.im, b.im)};
}
__device__ __forceinline__ C2 operator-(C2 a, C2 b) {
  return C2{f2_sub(a.re, b.re), f2_sub(a.im, b.im)};
}
__device__ __forceinline__ C2 mul_mi(C2 a) {  // -i a
  return C2{a.im, f2_sub(0ull, a.re)};
}
// a (wr + i wi) and a (wr - i wi), rounded as cmul(a, w) and cmul(a, cconj(w))
// are: the first product of a sum or difference is fused
__device__ __forceinline__ C2 mul_w(C2 a, float wr, float wi) {
  return C2{f2_fma(a.re, f2_dup(wr), f2_mul(a.im, f2_dup(-wi))),
            f2_fma(a.re, f2_dup(wi), f2_mul(a.im, f2_dup(wr)))};
}
__device__ __forceinline__ C2 mul_wc(C2 a, float wr, float wi) {
  return C2{f2_fma(a.re, f2_dup(wr), f2_mul(a.im, f2_dup(wi))),
            f2_fma(a.im, f2_dup(wr), f2_mul(a.re, f2_dup(-wi)))};
}

// cos and sin of 2 pi k / n at compile time (Taylor series in double)
constexpr double kTwoPi = 6.283185307179586476925286766559;
constexpr double ct_cos(int k, int n) {
  k %= n;
  if (2 * k > n) k = n - k;  // [0, pi]
  const bool neg = 4 * k > n;
  const double x = neg ? kTwoPi * (n - 2 * k) / (2.0 * n) : kTwoPi * k / n;  // [0, pi / 2]
  double t = 1.0, s = 1.0;
  for (int i = 1; i < 14; ++i) {
    t *= -x * x / ((2 * i - 1) * (2 * i));
    s += t;
  }
  return neg ? -s : s;
}
constexpr double ct_sin(int k, int n) {
  k %= n;
  const bool neg = 2 * k > n;
  if (neg) k = n - k;
  if (4 * k > n) {  // sin x = sin(pi - x)
    const double x = kTwoPi * (n - 2 * k) / (2.0 * n);
    double t = x, s = x;
    for (int i = 1; i < 14; ++i) {
      t *= -x * x / ((2 * i) * (2 * i + 1));
      s += t;
    }
    return neg ? -s : s;
  }
  const double x = kTwoPi * k / n;
  double t = x, s = x;
  for (int i = 1; i < 14; ++i) {
    t *= -x * x / ((2 * i) * (2 * i + 1));
    s += t;
  }
  return neg ? -s : s;
}
template <int K, int N>
struct Root {
  static constexpr float c = (float)ct_cos(K, N), s = (float)ct_sin(K, N);
};

__device__ __forceinline__ void dft3(C2 &a, C2 &b, C2 &c) {
  const C2 s = b + c, d = b - c;
  const f2 h = f2_dup(-0.5f), k = f2_dup(Root<1, 3>::s);
  const C2 e{f2_fma(s.re, h, a.re), f2_fma(s.im, h, a.im)};
  const C2 t{f2_fma(d.re, k, 0ull), f2_fma(d.im, k, 0ull)};
  a = a + s;
  b = C2{f2_add(e.re, t.im), f2_sub(e.im, t.re)};
  c = C2{f2_sub(e.re, t.im), f2_add(e.im, t.re)};
}
__device__ __forceinline__ void dft4(C2 &a, C2 &b, C2 &c, C2 &d) {
  const C2 p = a + c, q = a - c, r = b + d, s = mul_mi(b - d);
  a = p + r;
  b = q + s;
  c = p - r;
  d = q - s;
}

// cos and sin multiples of an odd P, unrolled at compile time
template <int P, int K, int R>
struct OddTerm {
  template <typename V>
  static __device__ __forceinline__ void run(const V &v, C2 &c, C2 &s) {
    OddTerm<P, K, R - 1>::run(v, c, s);
    const f2 cs = f2_dup(Root<(K * R) % P, P>::c), sn = f2_dup(Root<(K * R) % P, P>::s);
    c = C2{f2_fma(v[R].re, cs, c.re), f2_fma(v[R].im, cs, c.im)};
    s = R == 1 ? C2{f2_mul(v[P - R].re, sn), f2_mul(v[P - R].im, sn)}
               : C2{f2_fma(v[P - R].re, sn, s.re), f2_fma(v[P - R].im, sn, s.im)};
  }
};
template <int P, int K>
struct OddTerm<P, K, 0> {
  template <typename V>
  static __device__ __forceinline__ void run(const V &, C2 &, C2 &) {}
};
// Outputs K and P - K, and those of smaller K before them: with s_r = v_r +
// v_{P-r} (in v[r]) and d_r = v_r - v_{P-r} (in v[P-r]), o_K = C - i S and
// o_{P-K} = C + i S.
template <int P, int K>
struct OddOut {
  template <typename V, typename Put>
  static __device__ __forceinline__ void run(const V &v, const Put &put) {
    OddOut<P, K - 1>::run(v, put);
    C2 c = v[0], s = v[0];
    OddTerm<P, K, (P - 1) / 2>::run(v, c, s);
    put(K, C2{f2_add(c.re, s.im), f2_sub(c.im, s.re)});
    put(P - K, C2{f2_sub(c.re, s.im), f2_add(c.im, s.re)});
  }
};
template <int P>
struct OddOut<P, 0> {
  template <typename V, typename Put>
  static __device__ __forceinline__ void run(const V &, const Put &) {}
};

// P-point forward DFT of v; put(k, value) takes each output as it is ready.
template <int P>
struct Dft {
  template <typename Put>
  static __device__ __forceinline__ void run(C2 (&v)[P], const Put &put) {
    C2 o = v[0];
#pragma unroll
    for (int r = 1; r <= (P - 1) / 2; ++r) {
      const C2 s = v[r] + v[P - r];
      v[P - r] = v[r] - v[P - r];
      v[r] = s;
      o = o + s;
    }
    put(0, o);
    OddOut<P, (P - 1) / 2>::run(v, put);
  }
};
template <>
struct Dft<2> {
  template <typename Put>
  static __device__ __forceinline__ void run(C2 (&v)[2], const Put &put) {
    put(0, v[0] + v[1]);
    put(1, v[0] - v[1]);
  }
};
template <>
struct Dft<3> {
  template <typename Put>
  static __device__ __forceinline__ void run(C2 (&v)[3], const Put &put) {
    dft3(v[0], v[1], v[2]);
    put(0, v[0]);
    put(1, v[1]);
    put(2, v[2]);
  }
};
template <>
struct Dft<4> {
  template <typename Put>
  static __device__ __forceinline__ void run(C2 (&v)[4], const Put &put) {
    dft4(v[0], v[1], v[2], v[3]);
#pragma unroll
    for (int k = 0; k < 4; ++k) put(k, v[k]);
  }
};
template <>
struct Dft<8> {
  template <typename Put>
  static __device__ __forceinline__ void run(C2 (&v)[8], const Put &put) {
    dft4(v[0], v[2], v[4], v[6]);
    dft4(v[1], v[3], v[5], v[7]);
    constexpr float h = Root<1, 8>::c;
    v[3] = mul_w(v[3], h, -h);
    v[5] = mul_mi(v[5]);
    v[7] = mul_w(v[7], -h, -h);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      put(k, v[2 * k] + v[2 * k + 1]);
      put(k + 4, v[2 * k] - v[2 * k + 1]);
    }
  }
};
template <>
struct Dft<9> {
  template <typename Put>
  static __device__ __forceinline__ void run(C2 (&v)[9], const Put &put) {
#pragma unroll
    for (int b = 0; b < 3; ++b) dft3(v[b], v[3 + b], v[6 + b]);
    v[4] = mul_w(v[4], Root<1, 9>::c, -Root<1, 9>::s);
    v[5] = mul_w(v[5], Root<2, 9>::c, -Root<2, 9>::s);
    v[7] = mul_w(v[7], Root<2, 9>::c, -Root<2, 9>::s);
    v[8] = mul_w(v[8], Root<4, 9>::c, -Root<4, 9>::s);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      dft3(v[3 * k], v[3 * k + 1], v[3 * k + 2]);
#pragma unroll
      for (int j = 0; j < 3; ++j) put(k + 3 * j, v[3 * k + j]);
    }
  }
};
template <>
struct Dft<16> {
  template <typename Put>
  static __device__ __forceinline__ void run(C2 (&v)[16], const Put &put) {
#pragma unroll
    for (int b = 0; b < 4; ++b) dft4(v[b], v[4 + b], v[8 + b], v[12 + b]);
    // v[4 k + b]: multiply by W16^{k b}
    v[5] = mul_w(v[5], Root<1, 16>::c, -Root<1, 16>::s);
    v[6] = mul_w(v[6], Root<2, 16>::c, -Root<2, 16>::s);
    v[7] = mul_w(v[7], Root<3, 16>::c, -Root<3, 16>::s);
    v[9] = mul_w(v[9], Root<2, 16>::c, -Root<2, 16>::s);
    v[10] = mul_mi(v[10]);
    v[11] = mul_w(v[11], Root<6, 16>::c, -Root<6, 16>::s);
    v[13] = mul_w(v[13], Root<3, 16>::c, -Root<3, 16>::s);
    v[14] = mul_w(v[14], Root<6, 16>::c, -Root<6, 16>::s);
    v[15] = mul_w(v[15], Root<9, 16>::c, -Root<9, 16>::s);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      dft4(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
#pragma unroll
      for (int j = 0; j < 4; ++j) put(k + 4 * j, v[4 * k + j]);
    }
  }
};

__device__ __forceinline__ C2 pfa_ld(const float4 *buf, unsigned slot) {
  const ulonglong2 w = reinterpret_cast<const ulonglong2 *>(buf)[slot];
  return C2{w.x, w.y};
}
__device__ __forceinline__ void pfa_st(float4 *buf, unsigned slot, C2 v) {
  reinterpret_cast<ulonglong2 *>(buf)[slot] = make_ulonglong2(v.re, v.im);
}

// One prime-factor pass, in place.
template <int P, int MODE>
__device__ __forceinline__ void pfa_pass(float4 *buf, unsigned m, unsigned step) {
  const unsigned M = m / P;
  for (unsigned u = threadIdx.x; u < M; u += blockDim.x) {
    const unsigned c = P * u;
    C2 v[P];
    unsigned a = c;
#pragma unroll
    for (int i = 0; i < P; ++i) {
      v[i] = pfa_ld(buf, pfa_slot<MODE>(a));
      a = pfa_wrap(a + step, m);
    }
    Dft<P>::run(v, [&](int k, C2 o) { pfa_st(buf, pfa_slot<MODE>(pfa_wrap(c + k * M, m)), o); });
  }
}

template <int MODE>
__device__ __forceinline__ void pfa_pass_any(float4 *buf, const FftPlan &p, int ip) {
  const unsigned m = p.m, st = p.step[ip];
  switch (p.radix[ip]) {
    case 3: pfa_pass<3, MODE>(buf, m, st); break;
    case 5: pfa_pass<5, MODE>(buf, m, st); break;
    case 7: pfa_pass<7, MODE>(buf, m, st); break;
    case 9: pfa_pass<9, MODE>(buf, m, st); break;
    case 11: pfa_pass<11, MODE>(buf, m, st); break;
    case 13: pfa_pass<13, MODE>(buf, m, st); break;
    default:
      if (MODE == kFftEven) switch (p.radix[ip]) {
          case 2: pfa_pass<2, MODE>(buf, m, st); break;
          case 4: pfa_pass<4, MODE>(buf, m, st); break;
          case 8: pfa_pass<8, MODE>(buf, m, st); break;
          case 16: pfa_pass<16, MODE>(buf, m, st); break;
        }
  }
}

// Stockham passes (in -> out).  A pass of radix P has butterflies j (0 <= j <
// m/P) that read in[j + r m/P], twiddle input r by W_{Ns P}^{k r} with
// k = j mod Ns, and write out[(j / Ns) Ns P + k + r Ns]; Ns is the product of
// the radices done.  A group of two consecutive radices PA, PB runs both in
// registers: butterfly J (0 <= J < m / (PA PB)) reads in[J + i m/(PA PB)], and
// the PB butterflies J + b m/(PA PB) of the first pass give the inputs of PA
// butterflies of the second.  INV: conjugate twiddles, and the outputs of a
// DFT in reverse order.  PAD: one word after each 8 spreads the first passes'
// strides over the banks (even lengths, where two such buffers have room).
template <bool PAD>
__device__ __forceinline__ int stock_slot(int a) {
  return PAD ? a + (a >> 3) : a;
}

// A group from its inputs v[b + PB a] = in[J + (b + PB a) m/(PA PB)] on; put(index,
// value) takes the outputs.
template <int PA, int PB, bool INV, typename Put>
__device__ __forceinline__ void stock_group(C2 (&v)[PA * PB], int J, int m, int Ns, unsigned magic,
                                            const float2 *__restrict__ tw, const Put &put) {
  // J / Ns as a multiply-high: magic = ceil(2^32 / Ns) is exact for
  // J, Ns < 2^16 (the error J * (magic - 2^32/Ns) / 2^32 < 2^-16 <= 1/Ns).
  const int q = Ns > 1 ? (int)__umulhi((unsigned)J, magic) : J;
  const int k = J - q * Ns;
  if (Ns > 1) {
    const int st = m / (Ns * PA);
#pragma unroll
    for (int a = 1; a < PA; ++a) {
      // k a st < Ns PA (m / (Ns PA)) = m: no reduction needed
      const float2 t = __ldg(tw + k * a * st);
#pragma unroll
      for (int b = 0; b < PB; ++b) {
        C2 &x = v[b + PB * a];
        x = INV ? mul_wc(x, t.x, t.y) : mul_w(x, t.x, t.y);
      }
    }
  }
  if constexpr (PB == 1) {
    const int base = q * Ns * PA + k;
    Dft<PA>::run(v, [&](int i, C2 o) { put(base + (INV && i > 0 ? PA - i : i) * Ns, o); });
  } else {
#pragma unroll
    for (int b = 0; b < PB; ++b) {
      C2 w[PA];
#pragma unroll
      for (int a = 0; a < PA; ++a) w[a] = v[b + PB * a];
      Dft<PA>::run(w, [&](int i, C2 o) { v[b + PB * (INV && i > 0 ? PA - i : i)] = o; });
    }
    const int NA = Ns * PA, st = m / (NA * PB);
#pragma unroll
    for (int a = 0; a < PA; ++a) {
      const int kb = k + a * Ns;
      C2 w[PB];
      w[0] = v[PB * a];
#pragma unroll
      for (int b = 1; b < PB; ++b) {
        const float2 t = __ldg(tw + kb * b * st);
        w[b] = INV ? mul_wc(v[b + PB * a], t.x, t.y) : mul_w(v[b + PB * a], t.x, t.y);
      }
      const int base = q * NA * PB + kb;
      Dft<PB>::run(w, [&](int i, C2 o) { put(base + (INV && i > 0 ? PB - i : i) * NA, o); });
    }
  }
}
__device__ __forceinline__ unsigned stock_magic(int Ns) {
  return Ns > 1 ? (unsigned)((0x100000000ull + (unsigned)Ns - 1) / (unsigned)Ns) : 0u;
}

// A group over shared memory; put takes the outputs.
template <int PA, int PB, bool INV, bool PAD, typename Put>
__device__ __forceinline__ void stock_pass(const float4 *in, int m, int Ns,
                                           const float2 *__restrict__ tw, const Put &put) {
  constexpr int Q = PA * PB;
  const int M = m / Q;
  const unsigned magic = stock_magic(Ns);
  for (int J = threadIdx.x; J < M; J += blockDim.x) {
    C2 v[Q];
#pragma unroll
    for (int i = 0; i < Q; ++i) v[i] = pfa_ld(in, stock_slot<PAD>(J + i * M));
    stock_group<PA, PB, INV>(v, J, m, Ns, magic, tw, put);
  }
}

// Calls f(PA, PB as constants) for a group code.
template <typename F>
__device__ __forceinline__ void stock_by_code(int code, const F &f) {
  using std::integral_constant;
  switch (code) {
    case 2 + 16: f(integral_constant<int, 2>(), integral_constant<int, 1>()); break;
    case 3 + 16: f(integral_constant<int, 3>(), integral_constant<int, 1>()); break;
    case 4 + 16: f(integral_constant<int, 4>(), integral_constant<int, 1>()); break;
    case 5 + 16: f(integral_constant<int, 5>(), integral_constant<int, 1>()); break;
    case 7 + 16: f(integral_constant<int, 7>(), integral_constant<int, 1>()); break;
    case 11 + 16: f(integral_constant<int, 11>(), integral_constant<int, 1>()); break;
    case 13 + 16: f(integral_constant<int, 13>(), integral_constant<int, 1>()); break;
    case 4 + 32: f(integral_constant<int, 4>(), integral_constant<int, 2>()); break;
    case 3 + 48: f(integral_constant<int, 3>(), integral_constant<int, 3>()); break;
    default: break;
  }
}

// Groups first .. last-1 from `in` on, between the two buffers of p.swords
// words at buf; every group ends with a barrier.  Returns the buffer that
// holds the result.
template <bool INV, bool PAD>
__device__ __forceinline__ float4 *stock_passes(float4 *buf, float4 *in, const FftPlan &p,
                                                int first, int last) {
  int Ns = 1;
  for (int g = 0; g < last; ++g) {
    const int code = p.stock[g];
    if (g >= first) {
      float4 *out = in == buf ? buf + p.swords : buf;
      stock_by_code(code, [&](auto PA, auto PB) {
        stock_pass<decltype(PA)::value, decltype(PB)::value, INV, PAD>(
            in, p.m, Ns, p.tw_m, [&](int n, C2 o) { pfa_st(out, stock_slot<PAD>(n), o); });
      });
      __syncthreads();
      in = out;
    }
    Ns *= (code & 15) * (code >> 4);
  }
  return in;
}

// The complex transform of the points in buf (written before a barrier).
// Returns the buffer that holds the result: buf itself, or the second one of a
// Stockham length.  (The inverse transform is the forward one with real and
// imaginary parts exchanged on the way in and out.)
template <int MODE>
__device__ __forceinline__ float4 *fft_passes(float4 *buf, const FftPlan &p) {
  if constexpr (MODE == kFftStockham) {
    return stock_passes<false, false>(buf, buf, p, 0, p.nstock);
  } else {
    for (int ip = 0; ip < p.npass; ++ip) {
      pfa_pass_any<MODE>(buf, p, ip);
      __syncthreads();
    }
    return buf;
  }
}

// Bins k and m - k of the real transforms whose packed complex transform has
// the values a at k and b at m - k (both at 0 for k = 0): X[k] = E + W_n^k O and
// X[m-k] = conj(E - W_n^k O), E = (a + conj b) / 2, O = -i (a - conj b) / 2
// for both signals.
__device__ __forceinline__ void pfa_rfft_bins(C2 a, C2 b, float2 w, C2 &xk, C2 &xmk) {
  const f2 half = f2_dup(0.5f);
  const C2 e{f2_mul(half, f2_add(a.re, b.re)), f2_mul(half, f2_sub(a.im, b.im))};
  const C2 o{f2_mul(half, f2_add(a.im, b.im)), f2_mul(half, f2_sub(b.re, a.re))};
  const C2 t = {f2_fma(f2_dup(w.x), o.re, f2_mul(f2_dup(-w.y), o.im)),
                f2_fma(f2_dup(w.x), o.im, f2_mul(f2_dup(w.y), o.re))};
  xk = e + t;
  xmk = C2{f2_sub(e.re, t.re), f2_sub(t.im, e.im)};
}
// Z[k] and Z[m-k] of the inverse split from bins a = X[k] and b = X[m-k]:
// Z[k] = E + i O, Z[m-k] = conj(E) + i conj(O) with
// E = (a + conj b) / 2, O = conj(w) (a - conj b) / 2.
__device__ __forceinline__ void pfa_irfft_pre(C2 a, C2 b, float2 w, C2 &zk, C2 &zmk) {
  const f2 half = f2_dup(0.5f);
  const C2 e{f2_mul(half, f2_add(a.re, b.re)), f2_mul(half, f2_sub(a.im, b.im))};
  const C2 d{f2_mul(half, f2_sub(a.re, b.re)), f2_mul(half, f2_add(a.im, b.im))};
  const C2 o = mul_wc(d, w.x, w.y);
  zk = C2{f2_sub(e.re, o.im), f2_add(e.im, o.re)};
  zmk = C2{f2_add(e.re, o.im), f2_sub(o.re, e.im)};
}

}  // namespace qpsdm

// mlp.cu -- the learned traveltime / t* surrogate on 5th-generation tensor cores.
//
// Network: 5 inputs (padded to 16) -> 4 x 128 (SiLU) -> 2 outputs (padded to
// 16).  BF16 weights and activations, FP32 accumulation in tensor memory,
// FP32 master weights and Adam moments in global memory.
//
// Every layer is a tcgen05 tile product (tc.cuh) on BF16 operands in shared
// memory, weights [out][in], with the FP32 accumulator in tensor memory.  Tiles
// are held transposed: TMEM lanes are the 128 features, columns the samples,
// and activations are kept as [feature][sample], which the products read
// either way round.  Warp w reads TMEM lane quarter (w mod 4) -- the quarter a
// warp may access is fixed by its warp index; a thread's bias is one number.
//
// Inference: six teams of four warps per CTA work on six tiles of 64 samples at
// once, each with its own mbarrier, TMEM columns and activation buffer (a layer's
// output overwrites its input once the MMA that read it has completed), so
// teams' MMAs run while others are in their epilogues.  Each thread loads its
// inputs of the next tile while the current one is computed.  The
// special-function queue bounds it (512 tanh a sample, 16 a cycle per SM: 3.0 ms
// for 26 M samples).  It runs dry while teams wait for their MMAs together:
// with two teams of eight warps, 128 samples as TMEM lanes and a load per bias
// 5.96 ms, three teams and biases read four to a load 4.92 ms, now 4.08 ms.
//
// Training: one team of 16 warps per CTA, T = 64 or 128 samples to a tile, T / 4
// of them to a thread:
//   Z_l^T = W_l H_{l-1}^T     dH_{l-1}^T = W_l^T dZ_l^T     dW_l = dZ_l^T H_{l-1}
// A thread's bias is one number and its part of a bias gradient a sum over its
// own registers.  Backward works from what forward left in place: Z2 and Z3 in
// tensor memory, Z4 in registers, H1..H4 in shared memory (for T = 128 H4 lies
// where W2 is, which is read again from L2 for the last product).  dZ_l takes
// the buffer of H_l, whose last reader is done by then.
// Each CTA writes its gradients to its own slice of a global buffer (the first
// tile's are stored, further ones added: plain, no atomics); one kernel then
// sums the slices in a fixed order, does the Adam step and writes the BF16
// images, so training is deterministic.
//
// SiLU(z) = z sigma(z) = h + h tanh(h), h = z / 2, with the hardware FP32
// tanh (tanh.approx.f32, about 2^-11 relative, below the BF16 rounding of
// the stored activations).  (The packed f16x2 tanh would halve the
// special-function work of the epilogue, the inference kernel's limiter,
// but its error is no longer small against BF16.)
#include <cuda_bf16.h>
#include <math.h>

#include <algorithm>
#include <mutex>
#include <utility>
#include <vector>

#include "common.cuh"
#include "internal.h"
#include "qpsdm_engine.h"
#include "tc.cuh"

namespace qpsdm {

constexpr int kH = 128, kIn = 16, kOut = 16;
// FP32 parameter block offsets
constexpr int oW1 = 0, oB1 = oW1 + kH * kIn;
constexpr int oW2 = oB1 + kH, oB2 = oW2 + kH * kH;
constexpr int oW3 = oB2 + kH, oB3 = oW3 + kH * kH;
constexpr int oW4 = oB3 + kH, oB4 = oW4 + kH * kH;
constexpr int oW5 = oB4 + kH, oB5 = oW5 + kOut * kH;
constexpr int kParams = oB5 + kOut;  // 53776
constexpr int kSlice = kParams + 16;  // + loss sum and padding
// BF16 weight images in the core-matrix layout (bytes)
constexpr int sW1 = 0, sW2 = sW1 + kH * kIn * 2, sW3 = sW2 + kH * kH * 2;
constexpr int sW4 = sW3 + kH * kH * 2, sW5 = sW4 + kH * kH * 2;
constexpr int kWBytes = sW5 + kOut * kH * 2;  // 106496
constexpr int kHBytes = kH * kH * 2;          // a [128][128] block
// biases in shared memory: half biases of layers 1-4 (the SiLU argument is
// h = (z + b) / 2), then b5
constexpr int kBiasBytes = (4 * kH + kOut) * 4;  // 2112
constexpr int kGradThreads = 512;
// training shared memory map for tiles of T samples
template <int T>
struct GradMap {
  static constexpr int xb = T * kIn * 2, hb = T * kH * 2;
  static constexpr int X = kWBytes;        // [T][16] bf16
  static constexpr int Y = X + xb;         // dZ5, [T][16] bf16
  static constexpr int H1 = Y + xb;        // H1^T, then dZ1^T: [128][T] bf16
  static constexpr int H2 = H1 + hb;       // H2^T, then dZ2^T
  static constexpr int H3 = H2 + hb;       // H3^T, then dZ3^T
  static constexpr bool in_w2 = T > 64;    // H4 in place of W2
  static constexpr int H4 = in_w2 ? sW2 : H3 + hb;
  static constexpr int bias = H3 + (in_w2 ? 1 : 2) * hb;
  static constexpr int db = bias + kBiasBytes;     // fp32 bias-gradient partials [4][4 parts][128]
  static constexpr int db5 = db + 16 * kH * 4;     // of layer 5: [T / 32][16]
  static constexpr int loss = db5 + 4 * kOut * 4;  // fp32 loss partials [16 warps]
  static constexpr int bytes = loss + 64;          // 186,752 (T = 64), 223,616 (T = 128)
};
// inference shared memory map: weights, biases, then per team X and H^T of a
// tile; 1 KB behind the last (k_mlp_forward)
constexpr int kFwdTile = 64, kFwdTeams = 6, kFwdTeam = 128;
constexpr int kFwdTeamBytes = kFwdTile * (kIn + kH) * 2;
constexpr int fBias = kWBytes;
constexpr int fTeam0 = fBias + 2304;
constexpr int kFwdSmem = fTeam0 + kFwdTeams * kFwdTeamBytes + 1024;  // 220,416 bytes

struct MlpTileArgs {
  float in_scale[5], in_shift[5];  // features = (raw - shift) * scale
  float w_out[2];                  // loss weights of the two outputs
  float inv_batch;
};

__device__ __forceinline__ float tanh_hw(float x) {
  float y;
  asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// h = (z + b) / 2 -> SiLU(z + b)
__device__ __forceinline__ float silu_h(float h) { return fmaf(h, tanh_hw(h), h); }
// SiLU'(u) = s (1 + u (1 - s)), s = sigma(u) = (1 + tanh(u / 2)) / 2, h = u / 2
__device__ __forceinline__ float silu_grad_h(float h) {
  const float s = fmaf(0.5f, tanh_hw(h), 0.5f);
  return s * fmaf(2.0f * h, 1.0f - s, 1.0f);
}

// 8 bf16 of row r, columns c..c+7 of a K-major core-matrix buffer (rowlen K).
__device__ __forceinline__ void st_row8(uint8_t *buf, int r, int c, int K, const float *v) {
  __nv_bfloat162 p[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) p[i] = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
  *reinterpret_cast<uint4 *>(buf + tc::kmaj_off(r, c, K)) = *reinterpret_cast<uint4 *>(p);
}

// A group of threads synchronised by its own named barrier.
struct Team {
  uint32_t id, nthr;
  __device__ __forceinline__ void sync() const {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(nthr) : "memory");
  }
  // true on every thread of the team if p is true on any
  __device__ __forceinline__ bool any(bool p) const {
    uint32_t r;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.u32 p, %1, 0;\n\t"
        "bar.red.or.pred q, %2, %3, p;\n\t"
        "selp.u32 %0, 1, 0, q;\n\t}"
        : "=r"(r)
        : "r"((uint32_t)p), "r"(id), "r"(nthr)
        : "memory");
    return r != 0;
  }
};

// Position of a team thread: TMEM lane quarter, column part, tile row.
struct Role {
  int lane, quarter, part, row;
  uint32_t lane_base;  // TMEM address bits of the quarter's first lane
  __device__ __forceinline__ explicit Role(int t) {
    const int w = t >> 5;
    lane = t & 31;
    quarter = w & 3;
    part = w >> 2;
    row = quarter * 32 + lane;
    lane_base = (uint32_t)(quarter * 32) << 16;
  }
};

// Tile products of a team.  begin() orders the team's shared- and tensor-memory
// accesses before the products that the leader then adds and commits; finish()
// waits for them.  A wait that gave up sets *err at once and is known to the
// whole team at the next begin(), which returns false on every thread: no
// barrier of its own.
struct Gemm {
  Team team;
  uint64_t *bar;
  uint32_t phase;
  int *err;
  bool leader, failed;
  __device__ __forceinline__ bool begin() {
    tc::fence_smem_to_async();
    tc::fence_before_sync();
    const bool ok = !team.any(failed);
    tc::fence_after_sync();
    return ok;
  }
  // D (TMEM) = A * B^T.  a/b: core-matrix buffers with storage row length
  // a_len/b_len; *_mn = 1 reads the buffer transposed (MN-major).  K: the
  // reduction length.
  __device__ __forceinline__ void add(uint32_t d, const uint8_t *a, int a_len, int a_mn,
                                      const uint8_t *b, int b_len, int b_mn, int N,
                                      int K) const {
    const uint32_t a_lbo = a_mn ? (a_len / 8) * 128 : 128, a_sbo = a_mn ? 128 : (a_len / 8) * 128;
    const uint32_t b_lbo = b_mn ? (b_len / 8) * 128 : 128, b_sbo = b_mn ? 128 : (b_len / 8) * 128;
    tc::gemm_steps(d, tc::smem_u32(a), a_lbo, a_sbo, a_mn ? 2 * a_lbo : 256, tc::smem_u32(b),
                   b_lbo, b_sbo, b_mn ? 2 * b_lbo : 256, tc::idesc_bf16(128, N, a_mn, b_mn), K,
                   false);
  }
  __device__ __forceinline__ void commit() const { tc::mma_commit(bar); }
  __device__ __forceinline__ void finish() {
    if (!tc::mbar_wait(bar, phase, 1u << 30)) {
      failed = true;
      atomicExch(err, 1);
    }
    phase ^= 1u;
    tc::fence_after_sync();
  }
  // one product; false (on every thread) if an earlier wait gave up
  __device__ __forceinline__ bool run(uint32_t d, const uint8_t *a, int a_len, int a_mn,
                                      const uint8_t *b, int b_len, int b_mn, int N, int K) {
    if (!begin()) return false;
    if (leader) {
      add(d, a, a_len, a_mn, b, b_len, b_mn, N, K);
      commit();
    }
    finish();
    return true;
  }
};

// N accumulator columns [c0, c0+N) of this thread's row.
template <int N>
__device__ __forceinline__ void acc_ld(uint32_t acc, const Role &ro, int c0, float *v) {
  uint32_t r[N];
#pragma unroll
  for (int k = 0; k < N; k += 16) tc::tmem_ld16_nowait(acc + ro.lane_base + c0 + k, r + k);
#pragma unroll
  for (int k = 0; k < N; k += 16) tc::tmem_wait_ld_dep16(r + k);
#pragma unroll
  for (int i = 0; i < N; ++i) v[i] = __uint_as_float(r[i]);
}

// Normalised features of one sample into the X tile (zero padding to 16).
__device__ __forceinline__ void put_raw(uint8_t *sx, int row, const float *raw, bool live,
                                        const MlpTileArgs &ta) {
  float v[16];
#pragma unroll
  for (int j = 0; j < 16; ++j) v[j] = 0.0f;
  if (live)
#pragma unroll
    for (int j = 0; j < 5; ++j) v[j] = (raw[j] - ta.in_shift[j]) * ta.in_scale[j];
  st_row8(sx, row, 0, kIn, v);
  st_row8(sx, row, 8, kIn, v + 8);
}
__device__ __forceinline__ void load_raw(const float *__restrict__ x, int s, bool live,
                                         float *raw) {
#pragma unroll
  for (int j = 0; j < 5; ++j) raw[j] = live ? __ldg(x + (size_t)s * 5 + j) : 0.0f;
}
__device__ __forceinline__ void put_x(uint8_t *sx, int row, const float *__restrict__ x, int s,
                                      bool live, const MlpTileArgs &ta) {
  float raw[5];
  load_raw(x, s, live, raw);
  put_raw(sx, row, raw, live, ta);
}

// Copy weights (bf16 images) and biases (half biases for layers 1-4); NT threads.
template <int NT>
__device__ __forceinline__ void load_weights(uint8_t *sm, float *bias,
                                             const uint8_t *__restrict__ wimg,
                                             const float *__restrict__ params) {
  const uint4 *src = reinterpret_cast<const uint4 *>(wimg);
  uint4 *dst = reinterpret_cast<uint4 *>(sm);
  constexpr int kN = kWBytes / 16;
  uint4 w[(kN + NT - 1) / NT];
#pragma unroll
  for (int i = 0; i < (kN + NT - 1) / NT; ++i)
    if (i * NT + (int)threadIdx.x < kN) w[i] = src[i * NT + threadIdx.x];
  for (int i = threadIdx.x; i < 4 * kH; i += NT) {
    const int l = i / kH;
    bias[i] = 0.5f * params[(l == 0 ? oB1 : l == 1 ? oB2 : l == 2 ? oB3 : oB4) + i % kH];
  }
  if (threadIdx.x < kOut) bias[4 * kH + threadIdx.x] = params[oB5 + threadIdx.x];
#pragma unroll
  for (int i = 0; i < (kN + NT - 1) / NT; ++i)
    if (i * NT + (int)threadIdx.x < kN) dst[i * NT + threadIdx.x] = w[i];
}

// ---------------------------------------------------------------------------
// inference: y[n][2] from x[n][5]; six teams of 128 threads per CTA
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kFwdTeams * kFwdTeam, 1)
    k_mlp_forward(const uint8_t *__restrict__ wimg, const float *__restrict__ params,
                  const float *__restrict__ x, int nsamp, MlpTileArgs ta, float *__restrict__ y,
                  int *err) {
  constexpr int T = kFwdTile;
  extern __shared__ __align__(1024) uint8_t sm[];
  __shared__ uint64_t bars[kFwdTeams];
  __shared__ uint32_t tslot;
  const int tid = threadIdx.x, team_id = tid / kFwdTeam, t = tid % kFwdTeam;
  if (tid < 32) tc::tmem_alloc(&tslot, 512);  // T columns a team, a power of two
  if (tid == 0) {
    for (int i = 0; i < kFwdTeams; ++i) tc::mbar_init(&bars[i], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  float *bias = reinterpret_cast<float *>(sm + fBias);
  load_weights<kFwdTeams * kFwdTeam>(sm, bias, wimg, params);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const Role ro(t);
  uint8_t *sx = sm + fTeam0 + team_id * kFwdTeamBytes, *sh = sx + T * kIn * 2;
  const uint32_t acc = tslot + T * team_id;
  Gemm g{Team{1u + team_id, kFwdTeam}, &bars[team_id], 0u, err, t == 0, false};
  // H^T = SiLU(acc + b) of this thread's feature, 32 samples at a time
  auto epilogue = [&](float hb) {
#pragma unroll
    for (int c = 0; c < T; c += 32) {
      float v[32];
      acc_ld<32>(acc, ro, c, v);
#pragma unroll
      for (int i = 0; i < 32; ++i) v[i] = silu_h(fmaf(0.5f, v[i], hb));
#pragma unroll
      for (int k = 0; k < 32; k += 8) st_row8(sh, ro.row, c + k, T, v + k);
    }
  };
  const int ntiles = (nsamp + T - 1) / T, ahead = kFwdTeams * gridDim.x * T;
  // this thread's sample of its team's next tile, loaded one tile ahead
  const bool sample = ro.row < T;
  int tile = team_id * gridDim.x + blockIdx.x;
  float raw[5];
  load_raw(x, tile * T + ro.row, sample && tile < ntiles && tile * T + ro.row < nsamp, raw);
  for (; tile < ntiles; tile += kFwdTeams * gridDim.x) {
    const int s = tile * T + ro.row;
    const bool live = sample && s < nsamp;
    if (sample) {
      put_raw(sx, ro.row, raw, live, ta);
      load_raw(x, s + ahead, s < nsamp - ahead, raw);
    }
    if (!g.run(acc, sm + sW1, kIn, 0, sx, kIn, 0, T, kIn)) break;
    epilogue(bias[ro.row]);
    bool ok = true;
    for (int l = 1; l < 4 && ok; ++l) {
      ok = g.run(acc, sm + sW2 + (l - 1) * kH * kH * 2, kH, 0, sh, T, 1, T, kH);
      if (ok) epilogue(bias[l * kH + ro.row]);
    }
    // lanes are samples here; the upper 64 come from what lies behind H^T (at
    // most 1 KB past it) and are not used
    if (!ok || !g.run(acc, sh, T, 1, sm + sW5, kH, 0, kOut, kH)) break;
    if (sample) {
      float v[16];
      acc_ld<16>(acc, ro, 0, v);
      if (live && !g.failed) {
        y[(size_t)s * 2] = v[0] + bias[4 * kH];
        y[(size_t)s * 2 + 1] = v[1] + bias[4 * kH + 1];
      }
    }
  }
  tc::fence_before_sync();
  __syncthreads();
  if (tid < 32) tc::tmem_free(tslot, 512);
}

// ---------------------------------------------------------------------------
// training
// ---------------------------------------------------------------------------
// H^T = SiLU(z + b) of this thread's feature for samples c0..c0+N-1, into a
// [128][T] buffer.
template <int T, int N>
__device__ __forceinline__ void put_silu(const float *z, const Role &ro, float hb, uint8_t *out) {
  const int c0 = ro.part * N;
  float v[N];
#pragma unroll
  for (int i = 0; i < N; ++i) v[i] = silu_h(fmaf(0.5f, z[i], hb));
#pragma unroll
  for (int k = 0; k < N / 8; ++k) st_row8(out, ro.row, c0 + 8 * k, T, v + 8 * k);
}

// dZ^T = dH^T (acc) * SiLU'(z + b) into a [128][T] buffer; this thread's sum
// (pairs of pairs) into db[part][feature].  A dead sample's dH is 0.
template <int T, int N>
__device__ __forceinline__ void put_dz(const float *z, uint32_t acc, const Role &ro, float hb,
                                       uint8_t *out, float *db) {
  const int c0 = ro.part * N;
  float d[N];
  acc_ld<N>(acc, ro, c0, d);
#pragma unroll
  for (int i = 0; i < N; ++i) d[i] = d[i] * silu_grad_h(fmaf(0.5f, z[i], hb));
#pragma unroll
  for (int k = 0; k < N / 8; ++k) st_row8(out, ro.row, c0 + 8 * k, T, d + 8 * k);
#pragma unroll
  for (int o = N / 2; o > 0; o >>= 1)
#pragma unroll
    for (int i = 0; i < o; ++i) d[i] += d[i + o];
  db[ro.part * kH + ro.row] = d[0];
}

// Order of a weight block [128][K] in a gradient slice: [K / 4][128][4], so that a
// warp's rows (TMEM lanes) write 512 consecutive bytes.  Everything else
// (biases, W5, loss) is in parameter order.
__device__ __forceinline__ void put_grad4(float *gs, int off, int row, int c, const float *v,
                                          bool first) {
  float4 *p = reinterpret_cast<float4 *>(gs + off + c * kH + row * 4);
  float4 q = make_float4(v[0], v[1], v[2], v[3]);
  if (!first) {
    const float4 o = *p;
    q = make_float4(o.x + q.x, o.y + q.y, o.z + q.z, o.w + q.w);
  }
  *p = q;
}
// dW [128 out][128 in] tile (rows = TMEM lanes) into the slice, this
// thread's row and 32 columns.
__device__ __forceinline__ void put_grad128(uint32_t acc, const Role &ro, float *gs, int off,
                                            bool first) {
  float v[32];
  acc_ld<32>(acc, ro, ro.part * 32, v);
#pragma unroll
  for (int k = 0; k < 8; ++k) put_grad4(gs, off, ro.row, ro.part * 32 + 4 * k, v + 4 * k, first);
}

// x: [n][5], t: [n][2]; grads: [gridDim.x][kSlice]
//
// One tile is a chain of ten waits for tile products with the epilogues between
// them, and at the usual batch a CTA has one tile: latency bounds it.  So the
// chain is kept short (nothing is computed twice but Z1, products that are ready
// together are committed together), 512 threads share each epilogue, gradient
// tiles are written out while the next products run, and tiles of 64 samples
// are taken while one per SM is enough (grad_tile below).
// 8,192 samples: 85.7 us before, 33 us with the short chain on tiles of 128
// samples as rows, 16.7 us transposed on 128 tiles of 64 (25,000 cycles: 3,600
// to load the weights, 900 per wait for a 128-deep product, 2,000 per gradient tile).
template <int T>
__global__ void __launch_bounds__(kGradThreads, 1)
    k_mlp_grad(const uint8_t *__restrict__ wimg, const float *__restrict__ params,
               const float *__restrict__ x, const float *__restrict__ t, int nsamp,
               MlpTileArgs ta, float *__restrict__ grads, int *err) {
  using M = GradMap<T>;
  constexpr int N = T / 4;  // samples to a thread
  extern __shared__ __align__(1024) uint8_t sm[];
  __shared__ uint64_t bar;
  __shared__ uint32_t tslot;
  const int tid = threadIdx.x;
  // the update may be scheduled as soon as every CTA has started (it waits for
  // the end of this kernel before it reads a slice)
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  float *gs = grads + (size_t)blockIdx.x * kSlice;
  if (tid < 32) tc::tmem_alloc(&tslot, 512);
  if (tid == 0) {
    tc::mbar_init(&bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  float *bias = reinterpret_cast<float *>(sm + M::bias);
  load_weights<kGradThreads>(sm, bias, wimg, params);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  // tensor memory: accumulators A..D of 128 columns each
  const uint32_t tA = tslot, tB = tslot + 128, tC = tslot + 256, tD = tslot + 384;
  const Role ro(tid);
  const int c0 = ro.part * N;
  const bool sample = ro.part == 0 && ro.row < T;  // this thread reads and writes a sample
  const float hb1 = bias[ro.row], hb2 = bias[kH + ro.row], hb3 = bias[2 * kH + ro.row],
              hb4 = bias[3 * kH + ro.row];
  Gemm g{Team{1u, kGradThreads}, &bar, 0u, err, tid == 0, false};
  float *db = reinterpret_cast<float *>(sm + M::db), *db5 = reinterpret_cast<float *>(sm + M::db5);
  float loss = 0.0f;
  const int ntiles = (nsamp + T - 1) / T;
  for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const int s = tile * T + ro.row;
    const bool live = s < nsamp, first = tile == blockIdx.x;
    float t0 = 0.0f, t1 = 0.0f;
    if (sample) {
      put_x(sm + M::X, ro.row, x, s, live, ta);
      if (live) {
        t0 = __ldg(t + (size_t)s * 2);
        t1 = __ldg(t + (size_t)s * 2 + 1);
      }
    }
    // forward: Z1 in A, Z2 in B, Z3 in C, Z4 in registers, Y in A
    float z[N];
    if (!g.run(tA, sm + sW1, kIn, 0, sm + M::X, kIn, 0, T, kIn)) break;
    acc_ld<N>(tA, ro, c0, z);
    put_silu<T, N>(z, ro, hb1, sm + M::H1);
    if (!g.run(tB, sm + sW2, kH, 0, sm + M::H1, T, 1, T, kH)) break;
    acc_ld<N>(tB, ro, c0, z);
    put_silu<T, N>(z, ro, hb2, sm + M::H2);
    if (!g.run(tC, sm + sW3, kH, 0, sm + M::H2, T, 1, T, kH)) break;
    acc_ld<N>(tC, ro, c0, z);
    put_silu<T, N>(z, ro, hb3, sm + M::H3);
    if (!g.run(tD, sm + sW4, kH, 0, sm + M::H3, T, 1, T, kH)) break;
    acc_ld<N>(tD, ro, c0, z);
    put_silu<T, N>(z, ro, hb4, sm + M::H4);
    // Y: lanes are samples here; of a 64-sample tile the upper 64 lanes come
    // from what lies behind (at most 1 KB past H4, inside the block) and are not used
    if (!g.run(tA, sm + M::H4, T, 1, sm + sW5, kH, 0, kOut, kH)) break;
    // loss and dZ5 = dY (2 live columns of 16)
    if (sample) {
      float v[16], d5[16];
      acc_ld<16>(tA, ro, 0, v);
#pragma unroll
      for (int j = 0; j < 16; ++j) d5[j] = 0.0f;
      if (live) {
        const float e0 = v[0] + bias[4 * kH] - t0;
        const float e1 = v[1] + bias[4 * kH + 1] - t1;
        loss += ta.w_out[0] * e0 * e0 + ta.w_out[1] * e1 * e1;
        d5[0] = 2.0f * ta.w_out[0] * e0 * ta.inv_batch;
        d5[1] = 2.0f * ta.w_out[1] * e1 * ta.inv_batch;
      }
      st_row8(sm + M::Y, ro.row, 0, kOut, d5);
      st_row8(sm + M::Y, ro.row, 8, kOut, d5 + 8);
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        float a = d5[j];
        for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
        if (ro.lane == 0) db5[ro.quarter * kOut + j] = a;
      }
      if (ro.lane < kOut - 2) db5[ro.quarter * kOut + 2 + ro.lane] = 0.0f;
    }
    // layer 5: dH4^T = W5^T dZ5^T, dW5^T = H4^T dZ5 (rows = in)
    if (!g.begin()) break;
    if (g.leader) {
      g.add(tD, sm + sW5, kH, 1, sm + M::Y, kOut, 0, T, kOut);
      g.add(tA, sm + M::H4, T, 0, sm + M::Y, kOut, 1, kOut, T);
      g.commit();
    }
    g.finish();
    if (ro.part == 0) {
      float v[16];
      acc_ld<16>(tA, ro, 0, v);
#pragma unroll
      for (int j = 0; j < kOut; ++j) {
        float *p = gs + oW5 + j * kH + ro.row;
        *p = first ? v[j] : *p + v[j];
      }
    }
    put_dz<T, N>(z, tD, ro, hb4, sm + M::H4, db + 12 * kH);
    // layer 4
    if (!g.begin()) break;
    if (g.leader) {
      g.add(tD, sm + sW4, kH, 1, sm + M::H4, T, 1, T, kH);
      g.add(tA, sm + M::H4, T, 0, sm + M::H3, T, 0, kH, T);
      g.commit();
    }
    if constexpr (M::in_w2) {
      // W2 back from L2 (its place is free once these products are done)
      uint4 w2[kHBytes / 16 / kGradThreads];
#pragma unroll
      for (int i = 0; i < kHBytes / 16 / kGradThreads; ++i)
        w2[i] = __ldg(reinterpret_cast<const uint4 *>(wimg + sW2) + i * kGradThreads + tid);
      g.finish();
#pragma unroll
      for (int i = 0; i < kHBytes / 16 / kGradThreads; ++i)
        reinterpret_cast<uint4 *>(sm + sW2)[i * kGradThreads + tid] = w2[i];
    } else {
      g.finish();
    }
    acc_ld<N>(tC, ro, c0, z);
    put_dz<T, N>(z, tD, ro, hb3, sm + M::H3, db + 8 * kH);
    // layer 3; dW4 out meanwhile
    if (!g.begin()) break;
    if (g.leader) {
      g.add(tD, sm + sW3, kH, 1, sm + M::H3, T, 1, T, kH);
      g.add(tC, sm + M::H3, T, 0, sm + M::H2, T, 0, kH, T);
      g.commit();
    }
    put_grad128(tA, ro, gs, oW4, first);
    g.finish();
    acc_ld<N>(tB, ro, c0, z);
    put_dz<T, N>(z, tD, ro, hb2, sm + M::H2, db + 4 * kH);
    // layer 2 and Z1 again; dW3 out meanwhile
    if (!g.begin()) break;
    if (g.leader) {
      g.add(tD, sm + sW2, kH, 1, sm + M::H2, T, 1, T, kH);
      g.add(tA, sm + sW1, kIn, 0, sm + M::X, kIn, 0, T, kIn);
      g.add(tB, sm + M::H2, T, 0, sm + M::H1, T, 0, kH, T);
      g.commit();
    }
    put_grad128(tC, ro, gs, oW3, first);
    g.finish();
    acc_ld<N>(tA, ro, c0, z);
    put_dz<T, N>(z, tD, ro, hb1, sm + M::H1, db);
    // layer 1; dW2 and the bias gradients (parts in order) out meanwhile
    if (!g.begin()) break;
    if (g.leader) {
      g.add(tC, sm + M::H1, T, 0, sm + M::X, kIn, 1, kIn, T);
      g.commit();
    }
    put_grad128(tB, ro, gs, oW2, first);
    {
      const int l = tid / kH, c = tid % kH;  // 4 layers x 128
      const float *q = db + 4 * l * kH + c;
      float *p = gs + (l == 0 ? oB1 : l == 1 ? oB2 : l == 2 ? oB3 : oB4) + c;
      const float a = ((q[0] + q[kH]) + q[2 * kH]) + q[3 * kH];
      *p = first ? a : *p + a;
      if (tid < kOut) {
        float a5 = db5[tid];
        for (int i = 1; i < T / 32; ++i) a5 += db5[i * kOut + tid];
        float *p5 = gs + oB5 + tid;
        *p5 = first ? a5 : *p5 + a5;
      }
    }
    g.finish();
    if (ro.part == 0) {
      float v[16];
      acc_ld<16>(tC, ro, 0, v);
#pragma unroll
      for (int k = 0; k < 4; ++k) put_grad4(gs, oW1, ro.row, 4 * k, v + 4 * k, first);
    }
  }
  // loss sum of this CTA, in warp order
  for (int o = 16; o > 0; o >>= 1) loss += __shfl_xor_sync(0xffffffffu, loss, o);
  float *ls = reinterpret_cast<float *>(sm + M::loss);
  if (ro.lane == 0) ls[tid >> 5] = loss;
  tc::fence_before_sync();
  __syncthreads();
  if (tid == 0) {
    float a = 0.0f;
    for (int w = 0; w < T / 32; ++w) a += ls[w];  // the warps that had samples
    *reinterpret_cast<float4 *>(gs + kParams) = make_float4(a * ta.inv_batch, 0.0f, 0.0f, 0.0f);
  }
  if (tid < 32) tc::tmem_free(tslot, 512);
}

// BF16 core-matrix image of four weights of one row (row length K, columns c..c+3).
__device__ __forceinline__ void pack4(uint8_t *img, int r, int c, int K, const float4 &w) {
  __nv_bfloat162 h[2] = {__floats2bfloat162_rn(w.x, w.y), __floats2bfloat162_rn(w.z, w.w)};
  *reinterpret_cast<uint2 *>(img + tc::kmaj_off(r, c, K)) = *reinterpret_cast<uint2 *>(h);
}

// Four consecutive entries of a gradient slice: where they are in the
// parameters, and in the BF16 images (img < 0: a bias).
struct Slot {
  int p, img, r, c, K;
  __device__ __forceinline__ explicit Slot(int s) : p(s), img(-1), r(0), c(0), K(kH) {
    if (s < oB1) {
      K = kIn;
      img = sW1;
      r = (s % (4 * kH)) / 4;
      c = s / (4 * kH) * 4;
      p = oW1 + r * kIn + c;
    } else if (s >= oW5) {
      if (s < oB5) {
        img = sW5;
        r = (s - oW5) / kH;
        c = (s - oW5) % kH;
      }
    } else {
      const int l = (s - oW2) / (kH * kH + kH), e = (s - oW2) % (kH * kH + kH);
      if (s >= oW2 && e < kH * kH) {
        img = sW2 + l * kH * kH * 2;
        r = (e % (4 * kH)) / 4;
        c = e / (4 * kH) * 4;
        p = oW2 + l * (kH * kH + kH) + r * kH + c;
      }
    }
  }
};

struct AdamArgs {
  float lr, b1, b2, eps, c1, c2;
};
__device__ __forceinline__ void adam1(float &p, float &m, float &v, float g, float mask,
                                      const AdamArgs &a) {
  const float gi = g * mask;
  const float mi = a.b1 * m + (1.0f - a.b1) * gi;
  const float vi = a.b2 * v + (1.0f - a.b2) * gi * gi;
  m = mi;
  v = vi;
  p = (p - a.lr * (mi * a.c1) / (sqrtf(vi * a.c2) + a.eps)) * mask;
}

// Sum the per-CTA slices in a fixed order, four entries to a thread and four
// threads (consecutive quarters of the slices) to a sum.  ADAM:
// then Adam on the FP32 master weights (padded entries are kept at zero) and
// their BF16 images; only the loss goes to g.  Else the gradients go to g, in
// parameter order.  The slices come from L2, up to 16 loads in flight a thread:
// 64 slices (13.8 MB) with the update 6.7 us (9.0 us for 128), where the sum
// (one load in flight), Adam and packing took 18.8 + 6.9 + 4.5 us as three
// launches; one thread to a sum took 9.6.
constexpr int kUpdSums = 96, kUpdParts = 4;
template <bool ADAM>
__global__ void __launch_bounds__(kUpdSums * kUpdParts)
    k_mlp_update(const float *__restrict__ grads, int nslice, float *__restrict__ p,
                 float *__restrict__ m, float *__restrict__ v, const float *__restrict__ mask,
                 AdamArgs a, uint8_t *__restrict__ wimg, float *__restrict__ g) {
  __shared__ float4 sums[kUpdParts][kUpdSums];
  const int j = threadIdx.x % kUpdSums, part = threadIdx.x / kUpdSums;
  const int s = 4 * (blockIdx.x * kUpdSums + j);
  const Slot o(s);
  const bool mine = part == 0 && s < kParams;
  float4 k4 = make_float4(0.0f, 0.0f, 0.0f, 0.0f), p4 = k4, m4 = k4, v4 = k4, q = k4;
  if (ADAM && mine) {
    k4 = *reinterpret_cast<const float4 *>(mask + o.p);
    p4 = *reinterpret_cast<float4 *>(p + o.p);
    m4 = *reinterpret_cast<float4 *>(m + o.p);
    v4 = *reinterpret_cast<float4 *>(v + o.p);
  }
  // end of the gradient kernel: its slices, and its reads of p
  asm volatile("griddepcontrol.wait;" ::: "memory");
  // s == kParams: the loss, in the first of the slice's last 16 entries
  if (s <= kParams) {
    const int per = (nslice + kUpdParts - 1) / kUpdParts;
    const int c1 = min(nslice, (part + 1) * per);
    const float *gp = grads + s;
#pragma unroll 16
    for (int c = part * per; c < c1; ++c) {
      const float4 u = *reinterpret_cast<const float4 *>(gp + (size_t)c * kSlice);
      q = make_float4(q.x + u.x, q.y + u.y, q.z + u.z, q.w + u.w);
    }
  }
  sums[part][j] = q;
  __syncthreads();
  if (part != 0 || s > kParams) return;
#pragma unroll
  for (int i = 1; i < kUpdParts; ++i) {
    const float4 u = sums[i][j];
    q = make_float4(q.x + u.x, q.y + u.y, q.z + u.z, q.w + u.w);
  }
  if (s == kParams) {
    g[s] = q.x;
    return;
  }
  if (!ADAM) {
    *reinterpret_cast<float4 *>(g + o.p) = q;
    return;
  }
  adam1(p4.x, m4.x, v4.x, q.x, k4.x, a);
  adam1(p4.y, m4.y, v4.y, q.y, k4.y, a);
  adam1(p4.z, m4.z, v4.z, q.z, k4.z, a);
  adam1(p4.w, m4.w, v4.w, q.w, k4.w, a);
  *reinterpret_cast<float4 *>(m + o.p) = m4;
  *reinterpret_cast<float4 *>(v + o.p) = v4;
  *reinterpret_cast<float4 *>(p + o.p) = p4;
  if (o.img >= 0) pack4(wimg + o.img, o.r, o.c, o.K, p4);
}

// BF16 images of given weights (pads stay zero).
__global__ void k_mlp_pack(const float *__restrict__ p, uint8_t *__restrict__ wimg) {
  const int s = 4 * (blockIdx.x * blockDim.x + threadIdx.x);
  if (s >= kParams) return;
  const Slot o(s);
  if (o.img >= 0)
    pack4(wimg + o.img, o.r, o.c, o.K, *reinterpret_cast<const float4 *>(p + o.p));
}

}  // namespace qpsdm


// ---------------------------------------------------------------------------
// C ABI
// ---------------------------------------------------------------------------
using namespace qpsdm;

struct qpsdm_mlp {
  int device = 0, nsm = 0;
  float *p = nullptr, *m = nullptr, *v = nullptr, *g = nullptr, *mask = nullptr;
  float *slices = nullptr;
  uint8_t *wimg = nullptr;
  int *err = nullptr;
  int64_t step = 0;
  MlpTileArgs ta{};
  // one workspace of the table calls (surrogate.cu), kept between them
  std::mutex ws_mu;
  void *ws = nullptr;
  size_t ws_bytes = 0;
};

namespace qpsdm {

// A device workspace of at least `bytes` for a call that ends with its work
// done: the one the handle keeps if it is free and large enough, else a new
// one, before which a kept one that is too small is given back.
// mlp_put_workspace keeps it in the handle again (the larger of two when calls
// overlapped) or frees it.
void *mlp_take_workspace(qpsdm_mlp *h, size_t bytes, size_t *got) {
  void *p = nullptr;
  {
    std::lock_guard<std::mutex> lk(h->ws_mu);
    p = h->ws;
    *got = h->ws_bytes;
    h->ws = nullptr;
    h->ws_bytes = 0;
  }
  if (p && *got >= bytes) return p;
  cudaFree(p);
  *got = bytes;
  if (cudaMalloc(&p, bytes) == cudaSuccess) return p;
  cudaGetLastError();  // told by the result
  return nullptr;
}
void mlp_put_workspace(qpsdm_mlp *h, void *p, size_t bytes) {
  if (!p) return;
  {
    std::lock_guard<std::mutex> lk(h->ws_mu);
    if (bytes > h->ws_bytes) {
      std::swap(p, h->ws);
      h->ws_bytes = bytes;
    }
  }
  cudaFree(p);
}
int mlp_device(const qpsdm_mlp *h) { return h->device; }

}  // namespace qpsdm

constexpr int kUpdGrid = (kParams / 4 + 1 + kUpdSums - 1) / kUpdSums;

// Gradient slices of n samples: tiles of 64 samples while every tile has an SM
// of its own, since the epilogues of half a tile take half the time; else of
// 128, which read the weights and write a slice half as often.  A step of 4,096
// samples: 22.6 us with tiles of 64, 27.7 with 128; 8,192: 23.2 and 26.7;
// 9,472 (the last that fits): 24.6 and 26.7.
static int mlp_grad_tiles(const qpsdm_mlp *h, int n, bool *small) {
  const int t64 = (n + 63) / 64, t128 = (n + 127) / 128;
  *small = t64 <= h->nsm;
  return *small ? t64 : std::min(t128, h->nsm);
}
static int mlp_grad_launch(const qpsdm_mlp *h, const float *d_x, const float *d_t, int n,
                           cudaStream_t st) {
  MlpTileArgs ta = h->ta;
  ta.inv_batch = 1.0f / n;
  bool small;
  const int grid = mlp_grad_tiles(h, n, &small);
  if (small)
    k_mlp_grad<64><<<grid, kGradThreads, GradMap<64>::bytes, st>>>(h->wimg, h->p, d_x, d_t, n, ta,
                                                                   h->slices, h->err);
  else
    k_mlp_grad<128><<<grid, kGradThreads, GradMap<128>::bytes, st>>>(
        h->wimg, h->p, d_x, d_t, n, ta, h->slices, h->err);
  return grid;
}

extern "C" int qpsdm_mlp_create(int device, qpsdm_mlp **out) {
  if (!out) return QPSDM_EINVAL;
  *out = nullptr;
  cudaDeviceProp prop;
  if (cudaGetDeviceProperties(&prop, device) != cudaSuccess) return QPSDM_ECUDA;
  if (prop.major != 10 || prop.minor != 0) return QPSDM_ENOKERNEL;
  cudaSetDevice(device);
  auto *h = new qpsdm_mlp;
  h->device = device;
  h->nsm = prop.multiProcessorCount;
  bool ok = cudaMalloc(&h->p, sizeof(float) * kParams) == cudaSuccess &&
            cudaMalloc(&h->m, sizeof(float) * kParams) == cudaSuccess &&
            cudaMalloc(&h->v, sizeof(float) * kParams) == cudaSuccess &&
            cudaMalloc(&h->g, sizeof(float) * kSlice) == cudaSuccess &&
            cudaMalloc(&h->mask, sizeof(float) * kParams) == cudaSuccess &&
            cudaMalloc(&h->slices, sizeof(float) * kSlice * h->nsm) == cudaSuccess &&
            cudaMalloc(&h->wimg, kWBytes) == cudaSuccess &&
            cudaMalloc(&h->err, sizeof(int)) == cudaSuccess;
  if (!ok) {
    qpsdm_mlp_destroy(h);
    return QPSDM_ENOMEM;
  }
  cudaMemset(h->p, 0, sizeof(float) * kParams);
  cudaMemset(h->m, 0, sizeof(float) * kParams);
  cudaMemset(h->v, 0, sizeof(float) * kParams);
  cudaMemset(h->wimg, 0, kWBytes);
  cudaMemset(h->err, 0, sizeof(int));
  // trainable entries: input columns 0..4 of W1, output rows 0..1 of W5 and b5
  std::vector<float> mk(kParams, 1.0f);
  for (int r = 0; r < kH; ++r)
    for (int k = 5; k < kIn; ++k) mk[oW1 + r * kIn + k] = 0.0f;
  for (int r = 2; r < kOut; ++r) {
    for (int k = 0; k < kH; ++k) mk[oW5 + r * kH + k] = 0.0f;
    mk[oB5 + r] = 0.0f;
  }
  cudaMemcpy(h->mask, mk.data(), sizeof(float) * kParams, cudaMemcpyHostToDevice);
  for (int j = 0; j < 5; ++j) h->ta.in_scale[j] = 1.0f;
  h->ta.w_out[0] = h->ta.w_out[1] = 1.0f;
  if (cudaFuncSetAttribute(k_mlp_grad<64>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           GradMap<64>::bytes) != cudaSuccess ||
      cudaFuncSetAttribute(k_mlp_grad<128>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           GradMap<128>::bytes) != cudaSuccess ||
      cudaFuncSetAttribute(k_mlp_forward, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           kFwdSmem) != cudaSuccess) {
    qpsdm_mlp_destroy(h);
    return QPSDM_ECUDA;
  }
  *out = h;
  return QPSDM_OK;
}

extern "C" int qpsdm_mlp_destroy(qpsdm_mlp *h) {
  if (!h) return QPSDM_OK;
  cudaFree(h->p);
  cudaFree(h->m);
  cudaFree(h->v);
  cudaFree(h->g);
  cudaFree(h->mask);
  cudaFree(h->slices);
  cudaFree(h->wimg);
  cudaFree(h->err);
  cudaFree(h->ws);
  delete h;
  return QPSDM_OK;
}

extern "C" int qpsdm_mlp_param_count(void) { return kParams; }

extern "C" int qpsdm_mlp_set_params(qpsdm_mlp *h, const float *host_params) {
  if (!h || !host_params) return QPSDM_EINVAL;
  cudaSetDevice(h->device);
  std::vector<float> p(host_params, host_params + kParams), mk(kParams);
  cudaMemcpy(mk.data(), h->mask, sizeof(float) * kParams, cudaMemcpyDeviceToHost);
  for (int i = 0; i < kParams; ++i) p[i] *= mk[i];
  if (cudaMemcpy(h->p, p.data(), sizeof(float) * kParams, cudaMemcpyHostToDevice) != cudaSuccess)
    return QPSDM_ECUDA;
  cudaMemset(h->m, 0, sizeof(float) * kParams);
  cudaMemset(h->v, 0, sizeof(float) * kParams);
  h->step = 0;
  k_mlp_pack<<<kUpdGrid, kUpdSums>>>(h->p, h->wimg);
  return cudaDeviceSynchronize() == cudaSuccess ? QPSDM_OK : QPSDM_ECUDA;
}

extern "C" int qpsdm_mlp_get_params(qpsdm_mlp *h, float *host_params) {
  if (!h || !host_params) return QPSDM_EINVAL;
  cudaSetDevice(h->device);
  return cudaMemcpy(host_params, h->p, sizeof(float) * kParams, cudaMemcpyDeviceToHost) ==
                 cudaSuccess
             ? QPSDM_OK
             : QPSDM_ECUDA;
}

extern "C" int qpsdm_mlp_set_scaling(qpsdm_mlp *h, const float *in_shift, const float *in_scale,
                                     const float *out_weight) {
  if (!h || !in_shift || !in_scale || !out_weight) return QPSDM_EINVAL;
  for (int j = 0; j < 5; ++j) {
    h->ta.in_shift[j] = in_shift[j];
    h->ta.in_scale[j] = in_scale[j];
  }
  h->ta.w_out[0] = out_weight[0];
  h->ta.w_out[1] = out_weight[1];
  return QPSDM_OK;
}

// The update (or, without ADAM, the sum alone) behind its gradient kernel on
// the stream, launched programmatically: its CTAs start and load their
// parameters and moments while the last gradient CTAs run (k_mlp_grad writes none
// of those).  A step of 8,192 samples 23.6 -> 21.7 us, of 4,096 22.6 -> 20.5.
template <bool ADAM>
static cudaError_t mlp_update_launch(qpsdm_mlp *h, int nslice, const AdamArgs &a,
                                     cudaStream_t st) {
  cudaLaunchConfig_t c = {};
  c.gridDim = dim3(kUpdGrid);
  c.blockDim = dim3(kUpdSums * kUpdParts);
  c.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  c.attrs = at;
  c.numAttrs = 1;
  return cudaLaunchKernelEx(&c, k_mlp_update<ADAM>, (const float *)h->slices, nslice, h->p, h->m,
                            h->v, (const float *)h->mask, a, h->wimg, h->g);
}

static int mlp_check_err(qpsdm_mlp *h) {
  int e = 0;
  if (cudaMemcpy(&e, h->err, sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess)
    return QPSDM_ECUDA;
  return e ? QPSDM_ETIMEOUT : QPSDM_OK;
}

extern "C" int qpsdm_mlp_gradients(qpsdm_mlp *h, const float *d_x, const float *d_t, int n,
                                   float *host_grads, float *loss, void *stream) {
  if (!h || !d_x || !d_t || n <= 0) return QPSDM_EINVAL;
  cudaSetDevice(h->device);
  cudaStream_t st = (cudaStream_t)stream;
  const int grid = mlp_grad_launch(h, d_x, d_t, n, st);
  const cudaError_t ue = mlp_update_launch<false>(h, grid, AdamArgs{}, st);
  if (ue != cudaSuccess || cudaGetLastError() != cudaSuccess ||
      cudaStreamSynchronize(st) != cudaSuccess)
    return QPSDM_ECUDA;
  int rc = mlp_check_err(h);
  if (rc) return rc;
  if (host_grads)
    cudaMemcpy(host_grads, h->g, sizeof(float) * kParams, cudaMemcpyDeviceToHost);
  if (loss) cudaMemcpy(loss, h->g + kParams, sizeof(float), cudaMemcpyDeviceToHost);
  return QPSDM_OK;
}

extern "C" int qpsdm_mlp_train_step(qpsdm_mlp *h, const float *d_x, const float *d_t, int n,
                                    float lr, float *loss, void *stream) {
  if (!h || !d_x || !d_t || n <= 0 || !(lr > 0.0f)) return QPSDM_EINVAL;
  cudaSetDevice(h->device);
  cudaStream_t st = (cudaStream_t)stream;
  const int grid = mlp_grad_launch(h, d_x, d_t, n, st);
  h->step += 1;
  const float b1 = 0.9f, b2 = 0.999f;
  const float c1 = 1.0f / (1.0f - powf(b1, (float)h->step));
  const float c2 = 1.0f / (1.0f - powf(b2, (float)h->step));
  const cudaError_t ue = mlp_update_launch<true>(
      h, grid, AdamArgs{lr, b1, b2, 1e-8f, c1, c2}, st);
  if (ue != cudaSuccess || cudaGetLastError() != cudaSuccess) return QPSDM_ECUDA;
  if (loss) {
    if (cudaMemcpyAsync(loss, h->g + kParams, sizeof(float), cudaMemcpyDeviceToHost, st) !=
            cudaSuccess ||
        cudaStreamSynchronize(st) != cudaSuccess)
      return QPSDM_ECUDA;
    return mlp_check_err(h);
  }
  return QPSDM_OK;
}

extern "C" int qpsdm_mlp_forward(qpsdm_mlp *h, const float *d_x, int n, float *d_y,
                                 void *stream) {
  if (!h || !d_x || !d_y || n <= 0) return QPSDM_EINVAL;
  cudaSetDevice(h->device);
  // a tile to an SM before a second team has one
  const int ntiles = (n + kFwdTile - 1) / kFwdTile;
  const int grid = ntiles < h->nsm ? ntiles : h->nsm;
  k_mlp_forward<<<grid, kFwdTeams * kFwdTeam, kFwdSmem, (cudaStream_t)stream>>>(
      h->wimg, h->p, d_x, n, h->ta, d_y, h->err);
  return cudaGetLastError() == cudaSuccess ? QPSDM_OK : QPSDM_ECUDA;
}

extern "C" int qpsdm_mlp_status(qpsdm_mlp *h) {
  if (!h) return QPSDM_EINVAL;
  cudaSetDevice(h->device);
  if (cudaDeviceSynchronize() != cudaSuccess) return QPSDM_ECUDA;
  return mlp_check_err(h);
}

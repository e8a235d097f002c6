// Tensor-core kernels of the learned state-selection proposal's MLP
// (kMlpIn -> 256 -> 256 -> 1, ReLU; BF16 weights and activations, FP32
// accumulation in tensor memory).
//
// k_mlp_fwd: the whole forward pass of 128-row tiles in one persistent kernel.
//   W1 (32 KB) and W2 (128 KB) stay in shared memory for the CTA's lifetime in
//   the canonical K-major layout (tc.h). Per tile: the feature rows are staged
//   by cp.async; one thread issues the layer-1 MMAs (M 128, N 256, K 64) into
//   tensor-memory columns 0-255; the four warps read their 32 rows back
//   (tcgen05.ld), add the bias, apply ReLU, round to BF16 and write the hidden
//   tile to shared memory in two K halves of 128, each followed by its 8
//   layer-2 MMAs into columns 256-511; the layer-2 epilogue adds the bias,
//   applies ReLU and takes the dot product with w3 in FP32: the score. Thread t
//   of the CTA owns row t of the tile (tensor-memory lane t).
// k_gemm_tn: D = A * B^T for the weight gradients (split over K) and for the
//   layer-1 input gradient (masked by the ReLU of layer 1), cp.async stages
//   feeding tcgen05.mma.
// Every wait on the tensor core is bounded (tc::mbar_wait); a time-out sets
// the error flag, the CTA stops, frees its tensor memory and returns.
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <random>
#include <vector>

#include "context.h"
#include "mlp.h"
#include "tc.h"

namespace gp {
namespace {

constexpr int kTileM = 128;
constexpr uint32_t kSmemW1 = 0;
constexpr uint32_t kSmemW2 = kSmemW1 + kMlpHid * kMlpInP * 2;   // 32 KB
constexpr uint32_t kSmemX = kSmemW2 + kMlpHid * kMlpHid * 2;    // +128 KB
constexpr uint32_t kSmemH = kSmemX + kTileM * kMlpInP * 2;      // +16 KB
constexpr uint32_t kSmemB1 = kSmemH + kTileM * 128 * 2;         // +32 KB (one K half of the hidden tile)
constexpr uint32_t kSmemB2 = kSmemB1 + kMlpHid * 4;
constexpr uint32_t kSmemW3 = kSmemB2 + kMlpHid * 4;
constexpr uint32_t kSmemPart = kSmemW3 + kMlpHid * 4;  // the two halves' partial dot products
constexpr uint32_t kSmemBar = kSmemPart + 256 * 4;
constexpr uint32_t kSmemFwd = kSmemBar + 64;

// cp.async of a row-major BF16 matrix [rows][kext] (K contiguous, row stride ld
// elements) into a canonical K-major tile; rows at or beyond nvalid read zeros.
__device__ __forceinline__ void stage_kmajor(uint8_t* tile, const __nv_bfloat16* src, int rows, int kext, int ld,
                                             int nvalid, int k0, int kvalid) {
  const int chunks = rows * (kext >> 3);
  for (int c = threadIdx.x; c < chunks; c += blockDim.x) {
    // 8 rows of a chunk column side by side: 128 bytes of the tile, no bank conflicts
    const int u = c >> 3, r = u / (kext >> 3) * 8 + (c & 7), kc = u % (kext >> 3);
    const int k = k0 + kc * 8;
    const bool ok = r < nvalid && k < kvalid;
    const __nv_bfloat16* g = ok ? src + (size_t)r * ld + k : src;
    tc::cp_async16(tile + tc::kmajor_off(r, kc * 8, kext), g, ok ? 16u : 0u);
  }
}

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  const __nv_bfloat162 b = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&b);
}

constexpr int kFwdThreads = 256;  // warps w and w + 4 share tensor-memory lanes 32 (w % 4) .. + 31 (the tile's
                                  // rows) and split the columns of every epilogue step between them

__global__ void __launch_bounds__(kFwdThreads, 1) k_mlp_fwd(MlpFwdArgs a) {
  extern __shared__ __align__(1024) uint8_t sm[];
  uint64_t* bar = reinterpret_cast<uint64_t*>(sm + kSmemBar);
  uint32_t* tslot = reinterpret_cast<uint32_t*>(sm + kSmemBar + 8);
  int* abort_flag = reinterpret_cast<int*>(sm + kSmemBar + 12);
  float* b1s = reinterpret_cast<float*>(sm + kSmemB1);
  float* b2s = reinterpret_cast<float*>(sm + kSmemB2);
  float* w3s = reinterpret_cast<float*>(sm + kSmemW3);
  float* part = reinterpret_cast<float*>(sm + kSmemPart);
  const int tid = threadIdx.x, warp = tid >> 5;
  const int trow = tid & (kTileM - 1);  // the tile row (tensor-memory lane) this thread reads
  const int chalf = tid >> 7;           // which half of each epilogue step's columns it takes
  const int ntiles = (a.n + kTileM - 1) / kTileM;
  if ((int)blockIdx.x >= ntiles) return;

  if (warp == 0) tc::tmem_alloc(tslot, 512);
  if (tid == 0) {
    tc::mbar_init(bar, 1);
    tc::fence_mbar_init();
    *abort_flag = 0;
  }
  stage_kmajor(sm + kSmemW1, a.w1, kMlpHid, kMlpInP, kMlpInP, kMlpHid, 0, kMlpInP);
  stage_kmajor(sm + kSmemW2, a.w2, kMlpHid, kMlpHid, kMlpHid, kMlpHid, 0, kMlpHid);
  tc::cp_async_commit();
  for (int j = tid; j < kMlpHid; j += blockDim.x) {
    b1s[j] = a.b1[j];
    b2s[j] = a.b2[j];
    w3s[j] = a.w3[j];
  }
  const float b3 = a.b3[0];
  tc::cp_async_wait<0>();
  tc::fence_proxy_async();
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tbase = *tslot;
  const uint32_t lane_off = (uint32_t)((warp & 3) * 32) << 16;
  const uint32_t sW1 = tc::smem_u32(sm + kSmemW1), sW2 = tc::smem_u32(sm + kSmemW2);
  const uint32_t sX = tc::smem_u32(sm + kSmemX), sH = tc::smem_u32(sm + kSmemH);
  constexpr uint32_t idesc = tc::idesc_bf16(kTileM, kMlpHid);
  uint32_t phase = 0;

  auto wait_mma = [&]() {
    if (!tc::mbar_wait(bar, phase)) *abort_flag = 1;
    phase ^= 1u;
    __syncthreads();
    tc::fence_after_sync();
    return *abort_flag == 0;
  };

  for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const int r0 = tile * kTileM;
    const int row = r0 + trow;
    stage_kmajor(sm + kSmemX, a.x + (size_t)r0 * kMlpInP, kTileM, kMlpInP, kMlpInP, a.n - r0, 0, kMlpInP);
    tc::cp_async_commit();
    tc::cp_async_wait<0>();
    tc::fence_proxy_async();
    __syncthreads();
    if (tid == 0) {
      tc::fence_after_sync();
#pragma unroll
      for (int s = 0; s < kMlpInP / 16; ++s)
        tc::mma_bf16(tbase, tc::smem_desc(sX + s * 256, 128, (kMlpInP / 8) * 128),
                     tc::smem_desc(sW1 + s * 256, 128, (kMlpInP / 8) * 128), idesc, s > 0);
      tc::commit(bar);
    }
    if (!wait_mma()) break;
    bool ok = true;
    for (int h = 0; h < 2 && ok; ++h) {
      // layer-1 epilogue for hidden units [128 h, 128 h + 128): bias, ReLU, BF16;
      // this thread takes 64 of them
#pragma unroll 1
      for (int c = 0; c < 2; ++c) {
        const int c0 = chalf * 64 + c * 32;  // column within the half
        float v[32];
        tc::tmem_ld32(tbase + lane_off + h * 128 + c0, v);
        uint32_t p[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const int j = h * 128 + c0 + 2 * i;
          p[i] = tc::pack_bf16(fmaxf(v[2 * i] + b1s[j], 0.f), fmaxf(v[2 * i + 1] + b1s[j + 1], 0.f));
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const uint4 u = make_uint4(p[4 * q], p[4 * q + 1], p[4 * q + 2], p[4 * q + 3]);
          *reinterpret_cast<uint4*>(sm + kSmemH + tc::kmajor_off(trow, c0 + q * 8, 128)) = u;
          if (a.h1 && row < a.n)
            *reinterpret_cast<uint4*>(a.h1 + (size_t)row * kMlpHid + h * 128 + c0 + q * 8) = u;
        }
      }
      tc::fence_proxy_async();
      tc::fence_before_sync();
      __syncthreads();
      if (tid == 0) {
        tc::fence_after_sync();
#pragma unroll
        for (int s = 0; s < 8; ++s)
          tc::mma_bf16(tbase + 256, tc::smem_desc(sH + s * 256, 128, 16 * 128),
                       tc::smem_desc(sW2 + (h * 8 + s) * 256, 128, (kMlpHid / 8) * 128), idesc, h > 0 || s > 0);
        tc::commit(bar);
      }
      ok = wait_mma();
    }
    if (!ok) break;
    // layer-2 epilogue: bias, ReLU, dot with w3 in FP32 (this thread: 128 of the
    // 256 columns in order; the two halves are added below)
    float acc = 0.f;
#pragma unroll 1
    for (int c = chalf * 4; c < chalf * 4 + 4; ++c) {
      float v[32];
      tc::tmem_ld32(tbase + lane_off + 256 + c * 32, v);
      uint32_t p[16];
#pragma unroll
      for (int i = 0; i < 32; ++i) {
        const int j = c * 32 + i;
        v[i] = fmaxf(v[i] + b2s[j], 0.f);
        acc = fmaf(v[i], w3s[j], acc);
      }
      if (a.h2 && row < a.n) {
#pragma unroll
        for (int i = 0; i < 16; ++i) p[i] = tc::pack_bf16(v[2 * i], v[2 * i + 1]);
#pragma unroll
        for (int q = 0; q < 4; ++q)
          *reinterpret_cast<uint4*>(a.h2 + (size_t)row * kMlpHid + c * 32 + q * 8) =
              make_uint4(p[4 * q], p[4 * q + 1], p[4 * q + 2], p[4 * q + 3]);
      }
    }
    part[tid] = acc;
    tc::fence_before_sync();
    __syncthreads();
    if (chalf == 0 && row < a.n) a.score[row] = (part[trow] + part[trow + kTileM]) + b3;
  }
  if (*abort_flag && tid == 0) atomicExch(a.err, 1);
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 0) tc::tmem_free(tbase, 512);
}

// D = A * B^T, M tile 128, N tile NT, K blocks of 64 in cp.async stages.
// The K extents here are short (256, or a split of 2,048 rows): bound by the latency of
// the loads and by the epilogue. So some 192 KB are kept in flight, and a thread writes
// its row in 16-byte stores (the masked product of 16,384 rows: 76 us with two stages and
// stores of single elements, 21 now).
template <int NT>
constexpr int kGemmStages = NT == 256 ? 4 : 8;

template <int NT, int EPI>
__global__ void __launch_bounds__(128) k_gemm_tn(GemmArgs g) {
  extern __shared__ __align__(1024) uint8_t sm[];
  constexpr uint32_t kA = kTileM * 64 * 2, kB = NT * 64 * 2, kStage = kA + kB;
  constexpr int ST = kGemmStages<NT>;
  uint64_t* bar = reinterpret_cast<uint64_t*>(sm + ST * kStage);
  uint32_t* tslot = reinterpret_cast<uint32_t*>(bar + ST);
  const int tid = threadIdx.x, warp = tid >> 5;
  const bool second = EPI == 0 && (int)blockIdx.y * NT >= g.N;
  const int m0 = blockIdx.x * kTileM, n0 = blockIdx.y * NT - (second ? g.N : 0);
  const __nv_bfloat16* const ga = second ? g.a2 : g.a;
  const __nv_bfloat16* const gb = second ? g.b2 : g.b;
  const int N = second ? g.N2 : g.N;
  const int kbeg = blockIdx.z * g.kchunk, kend = min(g.K, kbeg + g.kchunk);
  const int nkb = kend > kbeg ? (kend - kbeg) / 64 : 0;
  constexpr uint32_t ncols = NT < 32 ? 32 : NT;
  if (warp == 0) tc::tmem_alloc(tslot, ncols);
  if (tid == 0) {
    for (int i = 0; i < ST; ++i) tc::mbar_init(&bar[i], 1);
    tc::fence_mbar_init();
  }
  // Chunks of 16 bytes, 8 rows of a chunk column side by side (128 bytes of the tile, no
  // bank conflicts): this thread takes the rows r, r + 16, ... at one k of every block.
  // With one warp per scheduler the address arithmetic counts, so it is kept out of
  // the loop: tiles and blocks are whole.
  const int r = (tid >> 6) * 8 + (tid & 7), k = (tid >> 3 & 7) * 8;
  const __nv_bfloat16* pa = ga + (size_t)(m0 + r) * g.lda + kbeg + k;
  const __nv_bfloat16* pb = gb + (size_t)(n0 + r) * g.ldb + kbeg + k;
  const size_t sa16 = (size_t)16 * g.lda, sb16 = (size_t)16 * g.ldb;
  uint8_t* const dst = sm + tc::kmajor_off(r, k, 64);
  auto load = [&](int kb) {  // in order; one group per block, empty past the last
    if (kb < nkb) {
      uint8_t* d = dst + (kb % ST) * kStage;
      const __nv_bfloat16* p = pa;
#pragma unroll
      for (int i = 0; i < kTileM / 16; ++i, p += sa16) tc::cp_async16(d + i * 2048, p, 16u);
      p = pb;
#pragma unroll
      for (int i = 0; i < NT / 16; ++i, p += sb16) tc::cp_async16(d + kA + i * 2048, p, 16u);
      pa += 64;
      pb += 64;
    }
    tc::cp_async_commit();
  };
#pragma unroll
  for (int kb = 0; kb < ST; ++kb) load(kb);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tbase = *tslot;
  constexpr uint32_t idesc = tc::idesc_bf16(kTileM, NT);
  bool late = false, stop = false;
  for (int kb = 0; kb < nkb; ++kb) {
    tc::cp_async_wait<ST - 2>();
    tc::fence_proxy_async();
    if ((stop = __syncthreads_or(late))) break;
    if (tid == 0) {
      tc::fence_after_sync();
      const uint32_t sa = tc::smem_u32(sm + (kb % ST) * kStage), sb = sa + kA;
#pragma unroll
      for (int s = 0; s < 4; ++s)
        tc::mma_bf16(tbase, tc::smem_desc(sa + s * 256, 128, 1024), tc::smem_desc(sb + s * 256, 128, 1024), idesc,
                     kb > 0 || s > 0);
      tc::commit(&bar[kb % ST]);
    }
    if (kb > 0) {  // the stage of block kb - 1, once its MMAs have read it
      const int next = kb - 1 + ST;
      if (next < nkb) late |= !tc::mbar_wait(&bar[(kb - 1) % ST], ((kb - 1) / ST) & 1u);
      load(next);
    }
  }
  // the last commit covers every MMA issued before it
  if (nkb > 0 && !stop)
    late |= !tc::mbar_wait(&bar[(nkb - 1) % ST], ((nkb - 1) / ST) & 1u);
  tc::cp_async_wait<0>();
  stop = __syncthreads_or(late);
  tc::fence_after_sync();
  const int row = m0 + tid;
  if (!stop) {
    const uint32_t lane_off = (uint32_t)(warp * 32) << 16;
#pragma unroll 1
    for (int c = 0; c < NT / 32; ++c) {
      float v[32];
      if (nkb > 0) {
        tc::tmem_ld32(tbase + lane_off + c * 32, v);
      } else {
#pragma unroll
        for (int i = 0; i < 32; ++i) v[i] = 0.f;
      }
      const int nb = n0 + c * 32;
      if (EPI == 0) {
        float4* o = reinterpret_cast<float4*>((second ? g.out2 : g.out_f) + ((size_t)blockIdx.z * g.M + row) * N + nb);
#pragma unroll
        for (int i = 0; i < 8; ++i) o[i] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
      } else {
        const uint4* mk = reinterpret_cast<const uint4*>(g.mask + (size_t)row * N + nb);
        uint4* o = reinterpret_cast<uint4*>(g.out_b + (size_t)row * N + nb);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const uint4 m = mk[i];
          uint32_t mw[4] = {m.x, m.y, m.z, m.w};
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const float2 h = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&mw[k]));
            const int q = 8 * i + 2 * k;
            mw[k] = pack_bf16(h.x > 0.f ? v[q] : 0.f, h.y > 0.f ? v[q + 1] : 0.f);
          }
          o[i] = make_uint4(mw[0], mw[1], mw[2], mw[3]);
        }
      }
    }
  }
  if (stop && tid == 0) atomicExch(g.err, 1);
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 0) tc::tmem_free(tbase, ncols);
}

// FP32 feature rows [n][kMlpIn] to zero-padded BF16 rows [rows][kMlpInP].
__global__ void k_feat_bf16(const float* __restrict__ x, int n, int rows, __nv_bfloat16* __restrict__ out) {
  const int64_t tot = (int64_t)rows * kMlpInP;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < tot; i += (int64_t)gridDim.x * blockDim.x) {
    const int r = (int)(i / kMlpInP), c = (int)(i % kMlpInP);
    out[i] = __float2bfloat16_rn(r < n && c < kMlpIn ? x[(size_t)r * kMlpIn + c] : 0.f);
  }
}

// Columns of 64 rows of a BF16 matrix: the products over rows read their operands
// with the rows contiguous. Thread j loads column j (a row of the matrix per request of
// the block) and writes its 64 values, 128 bytes, in eight stores.
constexpr int kColRows = 64;

__device__ __forceinline__ void load_column(const __nv_bfloat16* __restrict__ m, int ld, int rb, int j,
                                            uint32_t (&v)[kColRows / 2]) {
  const unsigned short* p = reinterpret_cast<const unsigned short*>(m) + (size_t)rb * ld + j;
#pragma unroll
  for (int i = 0; i < kColRows / 2; ++i) v[i] = p[(size_t)(2 * i) * ld] | (uint32_t)p[(size_t)(2 * i + 1) * ld] << 16;
}

__device__ __forceinline__ void store_column(__nv_bfloat16* __restrict__ out, int rows, int rb, int j,
                                             const uint32_t (&v)[kColRows / 2]) {
  uint4* o = reinterpret_cast<uint4*>(out + (size_t)j * rows + rb);
#pragma unroll
  for (int i = 0; i < kColRows / 8; ++i) o[i] = make_uint4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
}

__device__ __forceinline__ float bf_lo(uint32_t v) { return __uint_as_float(v << 16); }
__device__ __forceinline__ float bf_hi(uint32_t v) { return __uint_as_float(v & 0xffff0000u); }

// Columns of the per-block partial sums (hpart rows): dL/dw3 | dL/db2 | dL/db3,
// loss | dL/db1. They are added over the blocks in block order (k_step), so
// a training step gives the same parameters on every run.
constexpr int kHpW3 = 0, kHpB2 = kMlpHid, kHpB3 = 2 * kMlpHid, kHpLoss = 2 * kMlpHid + 1,
              kHpB1 = 2 * kMlpHid + 2, kHpCols = 3 * kMlpHid + 2;

// Loss head and the gradients it feeds, for the rows [64 blockIdx.x, + 64):
// p = sigmoid(score), loss = wt * BCE(p, y) / n, ds = (p - y) * wt / n;
// dz2[r][j] = ds * w3[j] where h2[r][j] > 0, as rows and as columns; the columns of
// h1; the block's sums of dL/dw3, dL/db2, dL/db3 and the loss go to its row of
// hpart. Thread j owns hidden unit j; a row's scalars are formed by one thread.
// Bound by the latency of its loads, 64 in flight per thread (16,384 rows: 42 us with
// a row per iteration and 18 for the two transposes after it, 12 now).
__global__ void __launch_bounds__(kMlpHid) k_bwd_head(
    const float* __restrict__ score, const float* __restrict__ y, const float* __restrict__ wt,
    const __nv_bfloat16* __restrict__ h1, const __nv_bfloat16* __restrict__ h2, const float* __restrict__ w3, int rows,
    float inv_n, __nv_bfloat16* __restrict__ dz2, __nv_bfloat16* __restrict__ dz2t, __nv_bfloat16* __restrict__ h1t,
    float* __restrict__ hpart) {
  __shared__ float dss[kColRows], lss[kColRows];
  const int j = threadIdx.x, rb = blockIdx.x * kColRows;
  uint32_t v[kColRows / 2];
  load_column(h2, kMlpHid, rb, j, v);
  const float w3j = w3[j];
  if (j < kColRows) {
    const float s = score[rb + j], yy = y[rb + j], ww = wt[rb + j];
    const float p = 1.f / (1.f + expf(-s));
    dss[j] = (p - yy) * ww * inv_n;
    lss[j] = ww * inv_n * (fmaxf(s, 0.f) - s * yy + log1pf(expf(-fabsf(s))));
  }
  __syncthreads();
  float gw3 = 0.f, gb2 = 0.f;
  unsigned short* o = reinterpret_cast<unsigned short*>(dz2) + (size_t)rb * kMlpHid + j;
#pragma unroll
  for (int i = 0; i < kColRows / 2; ++i) {
    const float h0 = bf_lo(v[i]), hh = bf_hi(v[i]), d0 = dss[2 * i], d1 = dss[2 * i + 1];
    const float z0 = h0 > 0.f ? d0 * w3j : 0.f, z1 = hh > 0.f ? d1 * w3j : 0.f;
    gw3 = fmaf(d0, h0, gw3);
    gb2 += z0;
    gw3 = fmaf(d1, hh, gw3);
    gb2 += z1;
    v[i] = pack_bf16(z0, z1);
    o[(size_t)(2 * i) * kMlpHid] = (unsigned short)(v[i] & 0xffffu);
    o[(size_t)(2 * i + 1) * kMlpHid] = (unsigned short)(v[i] >> 16);
  }
  store_column(dz2t, rows, rb, j, v);
  load_column(h1, kMlpHid, rb, j, v);
  store_column(h1t, rows, rb, j, v);
  float* row = hpart + (size_t)blockIdx.x * kHpCols;
  row[kHpW3 + j] = gw3;
  row[kHpB2 + j] = gb2;
  if (j < 2) {
    const float* t = j == 0 ? dss : lss;
    float acc = 0.f;
    for (int r = 0; r < kColRows; ++r) acc += t[r];
    row[j == 0 ? kHpB3 : kHpLoss] = acc;
  }
}

// For the rows [64 blockIdx.x, + 64): the columns of dz1 and of x, and the block's
// sums over rows of dz1 into its row of hpart (dL/db1), thread j per column.
__global__ void __launch_bounds__(kMlpHid) k_dz1_columns(const __nv_bfloat16* __restrict__ dz1,
                                                         const __nv_bfloat16* __restrict__ x, int rows,
                                                         __nv_bfloat16* __restrict__ dz1t,
                                                         __nv_bfloat16* __restrict__ xt, float* __restrict__ hpart) {
  const int j = threadIdx.x, rb = blockIdx.x * kColRows;
  uint32_t v[kColRows / 2];
  load_column(dz1, kMlpHid, rb, j, v);
  store_column(dz1t, rows, rb, j, v);
  float acc = 0.f;
#pragma unroll
  for (int i = 0; i < kColRows / 2; ++i) {
    acc += bf_lo(v[i]);
    acc += bf_hi(v[i]);
  }
  hpart[(size_t)blockIdx.x * kHpCols + kHpB1 + j] = acc;
  if (j < kMlpInP) {
    load_column(x, kMlpInP, rb, j, v);
    store_column(xt, rows, rb, j, v);
  }
}

// The end of a step, a thread per parameter (and one for the loss): the gradient, from
// the splits of the weight products or the blocks' sums, added in order; with lr > 0 the
// Adam update of the FP32 master and the BF16 copies that the GEMMs read (16,384 rows:
// 11 us, against 35 for a kernel per part).
struct StepArgs {
  const float* part1;  // [splits][256][64]
  const float* part2;  // [splits][256][256]
  const float* hpart;  // [blocks][kHpCols]
  int splits, blocks;
  float* grad;
  float* loss;
  float *p, *m, *v;
  __nv_bfloat16 *w1, *w2, *w2t;
  float lr, b1, b2, eps, c1, c2;
};

__device__ __forceinline__ float sum_strided(const float* __restrict__ p, int n, size_t stride) {
  float acc = 0.f;
#pragma unroll 16
  for (int z = 0; z < n; ++z) acc += p[z * stride];
  return acc;
}

__global__ void __launch_bounds__(256) k_step(StepArgs a) {
  const int i = blockIdx.x * 256 + threadIdx.x;
  if (i > kMlpParams) return;
  if (i == kMlpParams) {
    *a.loss = sum_strided(a.hpart + kHpLoss, a.blocks, kHpCols);
    return;
  }
  const bool is1 = i < kOffB1, is2 = i >= kOffW2 && i < kOffB2;
  float g;
  if (is1) g = sum_strided(a.part1 + i - kOffW1, a.splits, kMlpHid * kMlpInP);
  else if (is2) g = sum_strided(a.part2 + i - kOffW2, a.splits, kMlpHid * kMlpHid);
  else {
    const int col = i < kOffW2 ? kHpB1 + i - kOffB1
                    : i < kOffW3 ? kHpB2 + i - kOffB2
                    : i < kOffB3 ? kHpW3 + i - kOffW3 : kHpB3;
    g = sum_strided(a.hpart + col, a.blocks, kHpCols);
  }
  a.grad[i] = g;
  if (!(a.lr > 0.f)) return;  // no update with a NaN rate either, as on the host
  const float mi = a.b1 * a.m[i] + (1.f - a.b1) * g;
  const float vi = a.b2 * a.v[i] + (1.f - a.b2) * g * g;
  a.m[i] = mi;
  a.v[i] = vi;
  const float p = a.p[i] - a.lr * (mi / a.c1) / (sqrtf(vi / a.c2) + a.eps);
  a.p[i] = p;
  const __nv_bfloat16 b = __float2bfloat16_rn(p);
  if (is1) a.w1[i - kOffW1] = b;
  if (is2) {
    const int e = i - kOffW2;
    a.w2[e] = b;
    a.w2t[(size_t)(e % kMlpHid) * kMlpHid + e / kMlpHid] = b;
  }
}

__global__ void k_pack_weights(const float* __restrict__ p, __nv_bfloat16* __restrict__ w1,
                               __nv_bfloat16* __restrict__ w2, __nv_bfloat16* __restrict__ w2t) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < kMlpHid * kMlpHid; i += gridDim.x * blockDim.x) {
    if (i < kMlpHid * kMlpInP) w1[i] = __float2bfloat16_rn(p[kOffW1 + i]);
    const int r = i / kMlpHid, c = i % kMlpHid;
    const __nv_bfloat16 b = __float2bfloat16_rn(p[kOffW2 + i]);
    w2[i] = b;
    w2t[(size_t)c * kMlpHid + r] = b;
  }
}

}  // namespace

size_t mlp_fwd_smem() { return kSmemFwd; }

cudaError_t launch_mlp_fwd(const MlpFwdArgs& a, int grid, cudaStream_t s) {
  if (a.n <= 0) return cudaSuccess;
  const int ntiles = (a.n + kTileM - 1) / kTileM;
  grid = std::max(1, std::min(grid, ntiles));
  cudaError_t e = set_smem_limit_once<k_mlp_fwd>((int)kSmemFwd);
  if (e != cudaSuccess) return e;
  k_mlp_fwd<<<grid, kFwdThreads, kSmemFwd, s>>>(a);
  return cudaGetLastError();
}

template <int NT, int EPI>
static cudaError_t gemm_launch(const GemmArgs& g, int splits, cudaStream_t s) {
  constexpr size_t smem = kGemmStages<NT> * (kTileM * 64 * 2 + NT * 64 * 2) + 128;
  cudaError_t e = set_smem_limit_once<k_gemm_tn<NT, EPI>>((int)smem);
  if (e != cudaSuccess) return e;
  const dim3 grid((g.M + kTileM - 1) / kTileM, (g.N + g.N2) / NT, splits);
  k_gemm_tn<NT, EPI><<<grid, 128, smem, s>>>(g);
  return cudaGetLastError();
}

cudaError_t launch_gemm_tn(const GemmArgs& g, int NT, int epi, int splits, cudaStream_t s) {
  // whole tiles and blocks, rows of whole 16-byte chunks
  if (g.M % kTileM || g.N % NT || g.N2 % NT || g.K % 64 || g.kchunk % 64 || (g.lda & 7) || (g.ldb & 7))
    return cudaErrorInvalidValue;
  if (NT == 256 && epi == 1) return gemm_launch<256, 1>(g, splits, s);
  if (NT == 64 && epi == 0) return gemm_launch<64, 0>(g, splits, s);
  return cudaErrorInvalidValue;
}

}  // namespace gp

// ---- host side: parameters, forward and one training step ----
namespace gp {
namespace {

int mlp_ensure(Context& c) {
  MlpState& M = c.mlp;
  if (M.ready) return GP_OK;
  cudaError_t e;
  for (DevBuf* b : {&M.param, &M.m, &M.v, &M.grad})
    if ((e = b->ensure((size_t)kMlpParams * 4)) != cudaSuccess) return c.cuda_fail(e, "mlp alloc");
  if ((e = M.w1.ensure((size_t)kMlpHid * kMlpInP * 2)) != cudaSuccess) return c.cuda_fail(e, "mlp alloc");
  if ((e = M.w2.ensure((size_t)kMlpHid * kMlpHid * 2)) != cudaSuccess) return c.cuda_fail(e, "mlp alloc");
  if ((e = M.w2t.ensure((size_t)kMlpHid * kMlpHid * 2)) != cudaSuccess) return c.cuda_fail(e, "mlp alloc");
  if ((e = M.err.ensure(8)) != cudaSuccess) return c.cuda_fail(e, "mlp alloc");
  if ((e = M.loss.ensure(8)) != cudaSuccess) return c.cuda_fail(e, "mlp alloc");
  cudaMemsetAsync(M.m.ptr, 0, (size_t)kMlpParams * 4, c.stream);
  cudaMemsetAsync(M.v.ptr, 0, (size_t)kMlpParams * 4, c.stream);
  cudaMemsetAsync(M.err.ptr, 0, 8, c.stream);
  M.step = 0;
  M.ready = true;
  return GP_OK;
}

float* params(MlpState& M) { return M.param.as<float>(); }

void pack(Context& c) {
  MlpState& M = c.mlp;
  k_pack_weights<<<256, 256, 0, c.stream>>>(params(M), M.w1.as<__nv_bfloat16>(), M.w2.as<__nv_bfloat16>(),
                                            M.w2t.as<__nv_bfloat16>());
  c.prof.kernel_launches += 1;
}

}  // namespace

int mlp_rows(Context& c, int rows) {
  MlpState& M = c.mlp;
  if (rows <= M.cap_rows) return GP_OK;
  const size_t R = (size_t)rows;
  cudaError_t e;
  if ((e = M.x.ensure(R * kMlpInP * 2)) != cudaSuccess) return c.cuda_fail(e, "mlp rows");
  if ((e = M.xt.ensure(R * kMlpInP * 2)) != cudaSuccess) return c.cuda_fail(e, "mlp rows");
  for (DevBuf* b : {&M.y, &M.wt, &M.score})
    if ((e = b->ensure(R * 4)) != cudaSuccess) return c.cuda_fail(e, "mlp rows");
  for (DevBuf* b : {&M.h1, &M.h1t, &M.h2, &M.dz2, &M.dz2t, &M.dz1, &M.dz1t})
    if ((e = b->ensure(R * kMlpHid * 2)) != cudaSuccess) return c.cuda_fail(e, "mlp rows");
  M.cap_rows = rows;
  return GP_OK;
}

int check_mlp_err(Context& c, const char* what) {
  int32_t err = 0;
  cudaMemcpyAsync(&err, c.mlp.err.ptr, 4, cudaMemcpyDeviceToHost, c.stream);
  cudaError_t e = cudaStreamSynchronize(c.stream);
  if (e != cudaSuccess) return c.cuda_fail(e, what);
  if (err) {
    cudaMemsetAsync(c.mlp.err.ptr, 0, 4, c.stream);
    return (c.fail(GP_E_CUDA, std::string(what) + ": a tensor-core wait timed out"), GP_E_CUDA);
  }
  return GP_OK;
}

int mlp_forward_device(Context& c, const __nv_bfloat16* x, int n, float* score, __nv_bfloat16* h1, __nv_bfloat16* h2) {
  MlpState& M = c.mlp;
  MlpFwdArgs a;
  a.x = x;
  a.w1 = M.w1.as<__nv_bfloat16>();
  a.w2 = M.w2.as<__nv_bfloat16>();
  a.b1 = params(M) + kOffB1;
  a.b2 = params(M) + kOffB2;
  a.w3 = params(M) + kOffW3;
  a.b3 = params(M) + kOffB3;
  a.score = score;
  a.h1 = h1;
  a.h2 = h2;
  a.n = n;
  a.err = M.err.as<int>();
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaEvent_t ea;
  c.prof_begin(ea);
  cudaError_t e = launch_mlp_fwd(a, sms, c.stream);
  c.prof_end(ea, 3, (double)n);
  c.prof.kernel_launches += 1;
  return e == cudaSuccess ? GP_OK : c.cuda_fail(e, "mlp forward launch");
}

// One step over n rows already staged in M.x / M.y / M.wt (padded to rows).
int mlp_train_device(Context& c, int n, int rows, float lr, bool want_grad) {
  MlpState& M = c.mlp;
  cudaStream_t s = c.stream;
  auto bf = [](DevBuf& b) { return b.as<__nv_bfloat16>(); };
  int rc = mlp_forward_device(c, bf(M.x), rows, M.score.as<float>(), bf(M.h1), bf(M.h2));
  if (rc != GP_OK) return rc;
  const int hb = rows / kColRows;
  cudaError_t e;
  if ((e = M.hpart.ensure((size_t)hb * kHpCols * 4)) != cudaSuccess) return c.cuda_fail(e, "mlp partial");
  k_bwd_head<<<hb, kMlpHid, 0, s>>>(M.score.as<float>(), M.y.as<float>(), M.wt.as<float>(), bf(M.h1), bf(M.h2),
                                    params(M) + kOffW3, rows, 1.0f / (float)n, bf(M.dz2), bf(M.dz2t), bf(M.h1t),
                                    M.hpart.as<float>());
  // dL/dh1 = dz2 W2, masked by layer 1's ReLU: dz1 (rows x 256)
  GemmArgs ga{};
  ga.a = bf(M.dz2);
  ga.b = bf(M.w2t);
  ga.M = rows;
  ga.N = kMlpHid;
  ga.K = kMlpHid;
  ga.lda = ga.ldb = kMlpHid;
  ga.kchunk = kMlpHid;
  ga.out_b = bf(M.dz1);
  ga.mask = bf(M.h1);
  ga.err = M.err.as<int>();
  e = launch_gemm_tn(ga, 256, 1, 1, s);
  if (e != cudaSuccess) return c.cuda_fail(e, "mlp dH1 launch");
  k_dz1_columns<<<hb, kMlpHid, 0, s>>>(bf(M.dz1), bf(M.x), rows, bf(M.dz1t), bf(M.xt), M.hpart.as<float>());
  // weight gradients, split over rows: dW2 = dz2^T h1 and dW1 = dz1^T x in one launch, of
  // 128 x 64 tiles (ten CTAs per split; with tiles of 128 x 256 and a launch each, 16,384
  // rows ran on 16 SMs: 93 and 46 us, against 36 for both)
  const int kchunk = 2048;
  const int splits = (rows + kchunk - 1) / kchunk;
  if ((e = M.partial.ensure((size_t)splits * kMlpHid * (kMlpHid + kMlpInP) * 4)) != cudaSuccess)
    return c.cuda_fail(e, "mlp partial");
  float* part2 = M.partial.as<float>();
  float* part1 = part2 + (size_t)splits * kMlpHid * kMlpHid;
  GemmArgs gw{};
  gw.a = bf(M.dz2t);
  gw.b = bf(M.h1t);
  gw.M = kMlpHid;
  gw.N = kMlpHid;
  gw.K = rows;
  gw.lda = gw.ldb = rows;
  gw.kchunk = kchunk;
  gw.out_f = part2;
  gw.err = M.err.as<int>();
  gw.a2 = bf(M.dz1t);
  gw.b2 = bf(M.xt);
  gw.N2 = kMlpInP;
  gw.out2 = part1;
  if ((e = launch_gemm_tn(gw, 64, 0, splits, s)) != cudaSuccess) return c.cuda_fail(e, "mlp weight gradient launch");
  StepArgs st{};
  st.part1 = part1;
  st.part2 = part2;
  st.hpart = M.hpart.as<float>();
  st.splits = splits;
  st.blocks = hb;
  st.grad = M.grad.as<float>();
  st.loss = M.loss.as<float>();
  st.p = params(M);
  st.m = M.m.as<float>();
  st.v = M.v.as<float>();
  st.w1 = bf(M.w1);
  st.w2 = bf(M.w2);
  st.w2t = bf(M.w2t);
  st.lr = lr;
  if (lr > 0.f) {
    M.step++;
    st.b1 = 0.9f;
    st.b2 = 0.999f;
    st.eps = 1e-8f;
    st.c1 = 1.f - std::pow(st.b1, (float)M.step);
    st.c2 = 1.f - std::pow(st.b2, (float)M.step);
  }
  k_step<<<(kMlpParams + 256) / 256, 256, 0, s>>>(st);
  c.prof.kernel_launches += 5;
  (void)want_grad;
  return GP_OK;
}

}  // namespace gp

using gp::Context;

static Context* Cx(gp_ctx* c) { return reinterpret_cast<Context*>(c); }

extern "C" {

int32_t gp_mlp_param_count(void) { return gp::kMlpParams; }

int gp_mlp_init(gp_ctx* ctx, uint64_t seed) {
  if (!ctx) return GP_E_ARG;
  Context& c = *Cx(ctx);
  int rc = gp::mlp_ensure(c);
  if (rc != GP_OK) return rc;
  // He-uniform weights (fan-in of the 48 real features, then 256), zero biases;
  // the padded feature columns 48..63 of W1 stay zero.
  std::vector<float> p(gp::kMlpParams, 0.f);
  std::mt19937_64 g(seed);
  std::uniform_real_distribution<float> u(-1.f, 1.f);
  const float a1 = std::sqrt(6.f / gp::kMlpIn), a2 = std::sqrt(6.f / gp::kMlpHid), a3 = std::sqrt(3.f / gp::kMlpHid);
  for (int j = 0; j < gp::kMlpHid; ++j)
    for (int f = 0; f < gp::kMlpIn; ++f) p[gp::kOffW1 + j * gp::kMlpInP + f] = a1 * u(g);
  for (int i = 0; i < gp::kMlpHid * gp::kMlpHid; ++i) p[gp::kOffW2 + i] = a2 * u(g);
  for (int j = 0; j < gp::kMlpHid; ++j) p[gp::kOffW3 + j] = a3 * u(g);
  return gp_mlp_set_params(ctx, p.data());
}

int gp_mlp_set_params(gp_ctx* ctx, const float* params) {
  if (!ctx || !params) return GP_E_ARG;
  Context& c = *Cx(ctx);
  int rc = gp::mlp_ensure(c);
  if (rc != GP_OK) return rc;
  for (int j = 0; j < gp::kMlpHid; ++j)
    for (int f = gp::kMlpIn; f < gp::kMlpInP; ++f)
      if (params[gp::kOffW1 + j * gp::kMlpInP + f] != 0.f)
        return (c.fail(GP_E_ARG, "mlp: padded feature columns 48..63 of W1 must be zero"), GP_E_ARG);
  cudaMemcpyAsync(c.mlp.param.ptr, params, (size_t)gp::kMlpParams * 4, cudaMemcpyHostToDevice, c.stream);
  cudaMemsetAsync(c.mlp.m.ptr, 0, (size_t)gp::kMlpParams * 4, c.stream);
  cudaMemsetAsync(c.mlp.v.ptr, 0, (size_t)gp::kMlpParams * 4, c.stream);
  c.mlp.step = 0;
  gp::pack(c);
  cudaError_t e = cudaStreamSynchronize(c.stream);
  return e == cudaSuccess ? GP_OK : c.cuda_fail(e, "mlp set params");
}

int gp_mlp_get_params(gp_ctx* ctx, float* params) {
  if (!ctx || !params) return GP_E_ARG;
  Context& c = *Cx(ctx);
  if (!c.mlp.ready) return (c.fail(GP_E_STATE, "mlp: no parameters (gp_mlp_init)"), GP_E_STATE);
  cudaMemcpyAsync(params, c.mlp.param.ptr, (size_t)gp::kMlpParams * 4, cudaMemcpyDeviceToHost, c.stream);
  cudaError_t e = cudaStreamSynchronize(c.stream);
  return e == cudaSuccess ? GP_OK : c.cuda_fail(e, "mlp get params");
}

static int stage_rows(Context& c, int32_t n, const float* x, int& rows) {
  rows = (n + 127) / 128 * 128;
  int rc = gp::mlp_rows(c, rows);
  if (rc != GP_OK) return rc;
  gp::DevBuf& tmp = c.mlp.xf;
  cudaError_t e = tmp.ensure((size_t)n * gp::kMlpIn * 4);
  if (e != cudaSuccess) return c.cuda_fail(e, "mlp staging");
  cudaMemcpyAsync(tmp.ptr, x, (size_t)n * gp::kMlpIn * 4, cudaMemcpyHostToDevice, c.stream);
  gp::k_feat_bf16<<<512, 256, 0, c.stream>>>(tmp.as<float>(), n, rows, c.mlp.x.as<__nv_bfloat16>());
  c.prof.kernel_launches += 1;
  return GP_OK;
}

int gp_mlp_forward(gp_ctx* ctx, int32_t n, const float* x, float* score, float* h1, float* h2) {
  if (!ctx || n <= 0 || !x || !score) return GP_E_ARG;
  Context& c = *Cx(ctx);
  if (!c.mlp.ready) return (c.fail(GP_E_STATE, "mlp: no parameters (gp_mlp_init)"), GP_E_STATE);
  int rows = 0;
  int rc = stage_rows(c, n, x, rows);
  if (rc != GP_OK) return rc;
  gp::MlpState& M = c.mlp;
  // the hidden activations are written only when the caller asks for them
  rc = gp::mlp_forward_device(c, M.x.as<__nv_bfloat16>(), n, M.score.as<float>(),
                              h1 ? M.h1.as<__nv_bfloat16>() : nullptr, h2 ? M.h2.as<__nv_bfloat16>() : nullptr);
  if (rc != GP_OK) return rc;
  cudaMemcpyAsync(score, M.score.ptr, (size_t)n * 4, cudaMemcpyDeviceToHost, c.stream);
  std::vector<__nv_bfloat16> hb;
  if (h1 || h2) hb.resize((size_t)n * gp::kMlpHid);
  rc = gp::check_mlp_err(c, "mlp forward");
  if (rc != GP_OK) return rc;
  for (int k = 0; k < 2; ++k) {
    float* out = k ? h2 : h1;
    if (!out) continue;
    cudaMemcpyAsync(hb.data(), (k ? M.h2 : M.h1).ptr, hb.size() * 2, cudaMemcpyDeviceToHost, c.stream);
    if (cudaStreamSynchronize(c.stream) != cudaSuccess) return c.cuda_fail(cudaGetLastError(), "mlp forward");
    for (size_t i = 0; i < hb.size(); ++i) out[i] = __bfloat162float(hb[i]);
  }
  return GP_OK;
}

int gp_mlp_train_step(gp_ctx* ctx, int32_t n, const float* x, const float* y, const float* wt, float lr, float* loss,
                      float* grad) {
  if (!ctx || n <= 0 || !x || !y) return GP_E_ARG;
  Context& c = *Cx(ctx);
  if (!c.mlp.ready) return (c.fail(GP_E_STATE, "mlp: no parameters (gp_mlp_init)"), GP_E_STATE);
  int rows = 0;
  int rc = stage_rows(c, n, x, rows);
  if (rc != GP_OK) return rc;
  gp::MlpState& M = c.mlp;
  std::vector<float> yy(rows, 0.f), ww(rows, 0.f);
  for (int i = 0; i < n; ++i) {
    yy[i] = y[i];
    ww[i] = wt ? wt[i] : 1.f;
  }
  cudaMemcpyAsync(M.y.ptr, yy.data(), (size_t)rows * 4, cudaMemcpyHostToDevice, c.stream);
  cudaMemcpyAsync(M.wt.ptr, ww.data(), (size_t)rows * 4, cudaMemcpyHostToDevice, c.stream);
  rc = gp::mlp_train_device(c, n, rows, lr, grad != nullptr);
  if (rc != GP_OK) return rc;
  if (grad) cudaMemcpyAsync(grad, M.grad.ptr, (size_t)gp::kMlpParams * 4, cudaMemcpyDeviceToHost, c.stream);
  float l = 0.f;
  cudaMemcpyAsync(&l, M.loss.ptr, 4, cudaMemcpyDeviceToHost, c.stream);
  rc = gp::check_mlp_err(c, "mlp train step");
  if (rc != GP_OK) return rc;
  if (loss) *loss = l;
  return GP_OK;
}

}  // extern "C"

// The precision variant of the imputation forward-backward: FP32 or BF16
// checkpoints and an FP64 chunk log-likelihood.
//
// Same HMM, same per-site arithmetic and same division of the work as the full
// precision path (kernels_impute_warp.cu, after imputation_hmm.cpp:80-353):
// sequential chains keep the scaling factor of every site and a row per kRowSites
// sites, and k_impute_block forms the posteriors. What differs:
//   - The memory. Each haplotype is split at M (a multiple of 32, about np / 2). Both
//     chains run their own halves and keep checkpoints of them, then the other's half in
//     windows, each followed by its posteriors (ckpt_layout): 1/4 byte per site and state
//     in FP32, 1/16 in BF16, and the rows of two windows, against 1/2 for all rows. The
//     chains run as many sites one after another as without windows.
//   - The sums over states have another fixed tree (state k: lane k % 32 of virtual
//     warp (k / 32) % 8; j in order, lanes at distances 16 .. 1, virtual warps at 1,
//     2, 4), that of the AlphaSums whose logarithms make up the log-likelihood.
//   - With BF16 checkpoints, the forward messages on [0, M) and the backward ones on
//     [M, np) are those recomputed from a row rounded to BF16 at the start of each
//     block of 32 sites (k_ckpt_block, one CTA per block: its factors replace the
//     chain's there), and either chain goes on from a rounded row at M.
//     Either kernel is bound by its chain of dependent steps: a site per step, of which
//     the sum over 256 J states, its barrier and its five shuffles are most. A chain has
//     two warps, so that a lane's states are independent work within a step and the
//     barrier joins two warps only; with 256 threads and both half passes in sequence,
//     each a chain of its own, 32 haplotypes (400 - 1,200 states) at 150,000 sites took
//     65 ms a call, against 26.
//   - The FP64 chunk log-likelihood sum_l log AlphaSum_l (the reference keeps no such
//     value), from the AlphaSum of every site, off the chain.
#include <cuda_bf16.h>

#include <type_traits>

#include "internal.h"

namespace gp {
namespace {

constexpr int kCkptThreads = 64;

struct CkptArgs {
  const int32_t* __restrict__ order;
  const int32_t* __restrict__ npoly;
  const int32_t* __restrict__ nstates;
  const uint32_t* __restrict__ hvar;
  const float4* __restrict__ em;
  const float2* __restrict__ tr;
  const uint8_t* __restrict__ fl;
  const int64_t* __restrict__ row_off;
  float* __restrict__ rows;  // per haplotype as ckpt_layout says, its states at the end of each row
  float* __restrict__ fac;   // [2][n][32 WB]
  float* __restrict__ asum;  // [n][32 WB] AlphaSum of every site
  int n, L, WB, Kp;
  int windows, win;          // win < 0: the chains' own halves
};

// Partial sums: virtual warp v's lane at 32 v + 8 (lane & 3) + (lane >> 2), so that
// lane 4 v + r of either warp adds the eight lanes = r (mod 4) of v, distances 16, 8
// and 4, from two 16-byte loads.
struct CkptSmem {
  float red[2][256];
  float4 rec[1 + 4 * 32 + 1];  // emission of allele 0 and 1, t / K and 1 - t into the site
};

// Steps through the blocks b_first .. b_last (in the direction of the chain). Rows
// entering blocks of 16 go to `out`, the one of block r0 first; in the chain's own half
// (OWN) in BF16 mode, rows entering blocks of 32 to the checkpoints instead.
// SEG: one block, from its BF16 checkpoint. J: 256 (J - 1) < K <= 256 J. U: steps unrolled.
template <int J, bool FWD, bool SEG, bool BF16, bool OWN, int U>
__device__ __forceinline__ void ckpt_run(const CkptArgs& A, CkptSmem& S, const CkptLayout& lay, int t, int b_first,
                                         int b_last, float* out, int r0) {
  constexpr int NP = 2 * J;  // packed pairs of states: virtual warps (0, 1) and (2, 3) of the warp, per j
  const int np = A.npoly[t], K = A.nstates[t];
  const int tid = threadIdx.x, lane = tid & 31, wi = tid >> 5;
  const int Ks = lay.Ks;
  // state of pair p: 256 (p / 2) + k0 + 64 (p & 1) (+ 32)
  const int k0 = 128 * wi + lane;
  auto state = [&](int p, int h) { return 256 * (p >> 1) + k0 + 64 * (p & 1) + 32 * h; };
  out += Ks - K;
  float* const saved = A.rows + A.row_off[t] + lay.state + (FWD ? 0 : 2 * Ks);  // the chain's row and sum
  float* fac = A.fac + ((size_t)(FWD ? 0 : A.n) + t) * 32 * A.WB;
  const uint32_t* hv = A.hvar + (size_t)t * A.WB * A.Kp;
  __nv_bfloat16* ck = reinterpret_cast<__nv_bfloat16*>(A.rows + A.row_off[t]);
  const float4* E = A.em + (size_t)t * A.L;
  const float2* T = A.tr + (size_t)t * A.L;
  const uint8_t* F = A.fl + (size_t)t * A.L;
  constexpr int dir = FWD ? 1 : -1;

  float4 pe = make_float4(0.f, 0.f, 0.f, 0.f);
  auto load_recs = [&](int b) {
    const int l = (b << 5) + lane;
    if (wi != 0 || l >= np) return;
    const float4 e = E[l];
    const bool f = F[l] != 0;
    const float2 tt = FWD ? (l > 0 ? T[l - 1] : make_float2(0.f, 0.f)) : T[l];
    pe = make_float4(f ? 1.0f : e.x, f ? 1.0f : e.y, tt.x, tt.y);
  };
  bool ok[4];  // the last four states
  f2 exists[2];
#pragma unroll
  for (int i = 0; i < 4; ++i) ok[i] = state(NP - 2 + (i >> 1), i & 1) < K;
#pragma unroll
  for (int i = 0; i < 2; ++i) exists[i] = f2_pack(ok[2 * i] ? 1.f : 0.f, ok[2 * i + 1] ? 1.f : 0.f);
  auto has = [&](int p, int h) { return p < NP - 2 || ok[2 * (p - (NP - 2)) + h]; };
  uint32_t w[2 * NP], wn[2 * NP];
  auto load_words = [&](int b) {
#pragma unroll
    for (int p = 0; p < NP; ++p)
#pragma unroll
      for (int h = 0; h < 2; ++h) wn[2 * p + h] = has(p, h) ? hv[(size_t)b * A.Kp + state(p, h)] : 0u;
  };
  f2 x[NP];
  auto store_row = [&](int i) {
#pragma unroll
    for (int p = 0; p < NP; ++p) {
      float v[2];
      f2_unpack(x[p], v[0], v[1]);
#pragma unroll
      for (int h = 0; h < 2; ++h)
        if (has(p, h)) out[(size_t)(i - r0) * Ks + state(p, h)] = v[h];
    }
  };
  auto round_row = [&]() {
#pragma unroll
    for (int p = 0; p < NP; ++p) {
      float a, b;
      f2_unpack(x[p], a, b);
      x[p] = f2_pack(__bfloat162float(__float2bfloat16_rn(a)), __bfloat162float(__float2bfloat16_rn(b)));
    }
  };

  const int l_first = FWD ? b_first << 5 : min(np, (b_first + 1) << 5) - 1;
  const bool init = FWD ? l_first == 0 : l_first == np - 1;
  load_recs(b_first);
  if (wi == 0) S.rec[1 + (b_first & 3) * 32 + lane] = pe;
  load_words(b_first);
#pragma unroll
  for (int p = 0; p < NP; ++p) {
    float v[2] = {0.f, 0.f};
    if (!init) {
#pragma unroll
      for (int h = 0; h < 2; ++h)
        if (has(p, h)) v[h] = SEG ? __bfloat162float(ck[(size_t)b_first * Ks + state(p, h)]) : saved[state(p, h)];
    }
    x[p] = f2_pack(v[0], v[1]);
  }
  float acc = SEG || init ? 1.f : saved[Ks];
  __syncthreads();
  const int wofs = 8 * (lane & 3) + (lane >> 2);
  const ulonglong2* const rin = reinterpret_cast<const ulonglong2*>(&S.red[0][8 * lane]);
  int parity = 0;
  float keep = 0.f, keep_sum = 0.f;  // lane i: factor and sum of the block's site i
  int i = l_first & 31;
  uint32_t m = 1u << i;
  const float4* rp = nullptr;
  float4 rec = make_float4(1.f, 1.f, 0.f, 0.f);

  auto step = [&](auto init_tag) {
    constexpr bool INIT = decltype(init_tag)::value;
    const float fact1 = INIT ? 1.0f / (float)K : rec.z;
    const float fact2 = INIT ? 0.f : rec.w / acc;
    const f2 f1 = f2_pack(fact1, fact1), f2v = f2_pack(fact2, fact2);
    const float ex = rec.x, ey = rec.y;
    if (lane == i) keep = fact2;
    f2 q[2];
#pragma unroll
    for (int p = 0; p < NP; ++p) {
      const bool b0 = (w[2 * p] & m) != 0u, b1 = (w[2 * p + 1] & m) != 0u;
      f2 nx = f2_mul(f2_fma(x[p], f2v, f1), f2_pack(b0 ? ey : ex, b1 ? ey : ex));
      if (p >= NP - 2) nx = f2_mul(nx, exists[p - (NP - 2)]);  // absent states are multiplied by 0, others by 1
      q[p & 1] = p < 2 ? nx : f2_add(q[p & 1], nx);
      x[p] = nx;
    }
    float* ro = &S.red[0][parity + 128 * wi + wofs];
    f2_unpack(q[0], ro[0], ro[32]);
    f2_unpack(q[1], ro[64], ro[96]);
    i += dir;
    m = FWD ? m << 1 : m >> 1;
    rp += dir;
    rec = *rp;
    __syncthreads();
    const ulonglong2 a = rin[parity >> 2], c = rin[(parity >> 2) + 1];
    float v0, v1;
    f2_unpack(f2_add(f2_add(a.x, c.x), f2_add(a.y, c.y)), v0, v1);
    float v = __fadd_rn(v0, v1);
    v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, 2));
    v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, 1));
#pragma unroll
    for (int o = 4; o < 32; o <<= 1) v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, o));
    // AlphaSum = 1 at a flat first site, betaSum = 1 at a flat last site (imputation_hmm.cpp:156,285)
    acc = INIT && F[l_first] != 0 ? 1.0f : v;
    if (FWD && !SEG && lane == i - dir) keep_sum = acc;
    parity ^= 256;
  };

  for (int b = b_first;; b += dir) {
#pragma unroll
    for (int p = 0; p < 2 * NP; ++p) w[p] = wn[p];
    rp = &S.rec[1 + (b & 3) * 32 + i];
    rec = *rp;
    if (SEG && !init) rec.w = fac[(b << 5) + i];  // the chain's factor into the block, divided by acc = 1
    if (b != b_last) {
      load_recs(b + dir);
      load_words(b + dir);
    }
    if (BF16 && !SEG && !(init && b == b_first)) {
      if (OWN) {
#pragma unroll
        for (int p = 0; p < NP; ++p) {
          float v[2];
          f2_unpack(x[p], v[0], v[1]);
#pragma unroll
          for (int h = 0; h < 2; ++h)
            if (has(p, h)) ck[(size_t)b * Ks + state(p, h)] = __float2bfloat16_rn(v[h]);
        }
      } else if (FWD ? b == lay.mblk : b == lay.mblk - 1) {
        round_row();
      }
    }
    if (b == b_first && init) step(std::integral_constant<bool, true>());
    const int end = FWD ? min(np - (b << 5), 32) : -1;
    while (i != end) {
      const int part = i / kRowSites;
      if (!(BF16 && OWN) && (FWD ? i == part * kRowSites : i == (part + 1) * kRowSites - 1))
        store_row(b * (32 / kRowSites) + part);
      const int stop = FWD ? min(end, (part + 1) * kRowSites) : part * kRowSites - 1;
#pragma unroll U
      while (i != stop) step(std::integral_constant<bool, false>());
    }
    if (wi == 0) {
      fac[(b << 5) + lane] = keep;
      if (FWD && !SEG) A.asum[(size_t)t * 32 * A.WB + (b << 5) + lane] = keep_sum;
    }
    if (b == b_last) break;
    if (wi == 0) S.rec[1 + ((b + dir) & 3) * 32 + lane] = pe;
    i = FWD ? 0 : 31;
    m = FWD ? 1u : 1u << 31;
    __syncthreads();
  }
  if (!SEG && (FWD ? b_last < lay.nblk - 1 : b_last > 0)) {  // the next launch goes on from here
#pragma unroll
    for (int p = 0; p < NP; ++p) {
      float v[2];
      f2_unpack(x[p], v[0], v[1]);
#pragma unroll
      for (int h = 0; h < 2; ++h)
        if (has(p, h)) saved[state(p, h)] = v[h];
    }
    if (tid == 0) saved[Ks] = acc;
  }
}

// Both chains of every haplotype, over their own halves or a window of the other's: CTA
// 2 c forward, 2 c + 1 backward.
template <int J, bool BF16, bool OWN, int U>
__global__ void __launch_bounds__(kCkptThreads, 1) k_ckpt_chain(CkptArgs A) {
  __shared__ CkptSmem S;
  const int t = A.order[blockIdx.x >> 1];
  const bool fwd = (blockIdx.x & 1) == 0;
  if (A.npoly[t] == 0 || A.nstates[t] == 0) return;
  const CkptLayout lay = ckpt_layout(A.npoly[t], A.nstates[t], BF16, A.windows);
  int lo = fwd ? 0 : lay.mblk, hi = fwd ? lay.mblk : lay.nblk;
  if (!OWN) ckpt_window(lay, fwd ? 0 : 1, A.win, lo, hi);
  if (lo >= hi) return;
  float* out = A.rows + A.row_off[t] + (OWN ? 0 : ckpt_window_rows(lay, fwd ? 0 : 1, A.win));
  const int r0 = OWN ? 0 : lo * (32 / kRowSites);
  if (fwd) ckpt_run<J, true, false, BF16, OWN, U>(A, S, lay, t, lo, hi - 1, out, r0);
  else ckpt_run<J, false, false, BF16, OWN, U>(A, S, lay, t, hi - 1, lo, out, r0);
}

// The rows of the other direction for one block of the window, from its BF16 checkpoint.
// blockIdx.x: the blocks in [M, np), then as many in [0, M); haplotype order[blockIdx.y].
template <int J>
__global__ void __launch_bounds__(kCkptThreads, 1) k_ckpt_block(CkptArgs A) {
  __shared__ CkptSmem S;
  const int t = A.order[blockIdx.y];
  if (A.npoly[t] == 0 || A.nstates[t] == 0) return;
  const CkptLayout lay = ckpt_layout(A.npoly[t], A.nstates[t], true, A.windows);
  const int per = gridDim.x / 2, half = (int)blockIdx.x >= per;
  int lo, hi;
  ckpt_window(lay, half, A.win, lo, hi);
  const int b = lo + (int)blockIdx.x - half * per;
  if (b >= hi) return;
  const int r0 = lo * (32 / kRowSites);
  float* out = A.rows + A.row_off[t] + ckpt_window_rows(lay, half, A.win) +
               (int64_t)(half ? lay.wlen1 : lay.wlen0) * (32 / kRowSites) * lay.Ks;
  if (half) ckpt_run<J, true, true, true, false, 1>(A, S, lay, t, b, b, out, r0);
  else ckpt_run<J, false, true, true, false, 1>(A, S, lay, t, b, b, out, r0);
}

// Sum of log AlphaSum over the sites of haplotype blockIdx.x, in FP64.
__global__ void __launch_bounds__(256) k_ckpt_loglik(const float* __restrict__ asum, const int32_t* __restrict__ npoly,
                                                     int WB, double* __restrict__ loglik) {
  __shared__ double part[256];
  const int t = blockIdx.x;
  double s = 0.0;
  for (int l = threadIdx.x; l < npoly[t]; l += 256) s += log((double)asum[(size_t)t * 32 * WB + l]);
  part[threadIdx.x] = s;
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if (threadIdx.x < o) part[threadIdx.x] += part[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) loglik[t] = part[0];
}

}  // namespace

static CkptArgs ckpt_args(ImputeWork& w, int windows, int win, float* asum, int first) {
  CkptArgs a;
  a.order = w.order.as<int32_t>() + first;
  a.npoly = w.npoly.as<int32_t>();
  a.nstates = w.nstates.as<int32_t>();
  a.hvar = w.hvar.as<uint32_t>();
  a.em = w.em.as<float4>();
  a.tr = w.tr.as<float2>();
  a.fl = w.fl.as<uint8_t>();
  a.row_off = w.row_off.as<int64_t>();
  a.rows = w.rows.as<float>();
  a.fac = w.fac.as<float>();
  a.asum = asum;
  a.n = w.n;
  a.L = w.L;
  a.WB = w.WB;
  a.Kp = w.Kp;
  a.windows = windows;
  a.win = win;
  return a;
}

#define GP_EACH_J(M) M(1) M(2) M(3) M(4) M(5) M(6) M(7) M(8)

// few: the batch's chains have an SM each. Their steps are then unrolled by four: a step is latency, and the loop's own
// instructions go (one haplotype at K = 600 11.6 -> 11.3 ms, 32 at K 400-1,200 18.3 -> 17.9). Where chains of
// mixed classes share SMs it costs a third (256: 31 -> 41 ms).
int launch_ckpt_chain(int J, bool bf16, bool few, int windows, int win, ImputeWork& w, float* asum, cudaStream_t s,
                      int first, int count) {
  const CkptArgs a = ckpt_args(w, windows, win, asum, first);
#define GP_CK1(JJ, UU)                                                                           \
  if (bf16 && win < 0) k_ckpt_chain<JJ, true, true, UU><<<2 * count, kCkptThreads, 0, s>>>(a);   \
  else if (bf16) k_ckpt_chain<JJ, true, false, UU><<<2 * count, kCkptThreads, 0, s>>>(a);        \
  else if (win < 0) k_ckpt_chain<JJ, false, true, UU><<<2 * count, kCkptThreads, 0, s>>>(a);     \
  else k_ckpt_chain<JJ, false, false, UU><<<2 * count, kCkptThreads, 0, s>>>(a);
#define GP_CK(JJ)         \
  case JJ:                \
    if (few) {            \
      GP_CK1(JJ, 4)       \
    } else {              \
      GP_CK1(JJ, 1)       \
    }                     \
    return GP_OK;
  switch (J) {
    GP_EACH_J(GP_CK)
    default: return GP_E_ARG;
  }
#undef GP_CK
#undef GP_CK1
}

int launch_ckpt_window(int J, bool bf16, int windows, int win, int wlen, ImputeWork& w, float* hp, cudaStream_t s,
                       int first, int count) {
  if (bf16 && wlen > 0) {
    const CkptArgs a = ckpt_args(w, windows, win, nullptr, first);
#define GP_CK(JJ) \
  case JJ: k_ckpt_block<JJ><<<dim3(2 * wlen, count), kCkptThreads, 0, s>>>(a); break;
    switch (J) {
      GP_EACH_J(GP_CK)
      default: return GP_E_ARG;
    }
#undef GP_CK
  }
  return launch_ckpt_posteriors(bf16, windows, win, wlen, w, hp, s, first, count);
}
#undef GP_EACH_J

void launch_ckpt_loglik(ImputeWork& w, const float* asum, double* loglik, cudaStream_t s) {
  k_ckpt_loglik<<<w.n, 256, 0, s>>>(asum, w.npoly.as<int32_t>(), w.WB, loglik);
}

}  // namespace gp

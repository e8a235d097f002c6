// Imputation HMM forward-backward: sequential chains that keep a row every 16
// sites, and a parallel pass over the blocks of 16 that forms the posteriors.
//
// The haploid Li-Stephens recursion (phase/src/models/imputation_hmm.cpp:143-416)
// is sequential over sites only through one number a site: the sum over all K
// states that scales the next site's factor (1 - t) / sum. Given those factors,
// every state's recursion runs by itself. So
//   k_impute_chain  runs both directions of a haplotype, each over all its sites,
//                   as two concurrent chains; it keeps the factor of every site
//                   and the row entering every block of 16 sites;
//   k_impute_block  runs one block of one haplotype per CTA: each thread repeats
//                   its states' forward steps from the kept row into registers and
//                   then the backward steps, multiplies the two and sums. The steps
//                   are the chain's own operations on the same numbers, so the
//                   rows it forms are the chain's, bit for bit.
// Measured, both kernels (K = 1,000, 62,700 polymorphic sites): one haplotype 11.6 ms,
// 256 haplotypes 23.6; with every row stored and read back by the chains, split in
// the middle of the haplotype, 16.3 and 33 ms.
// Nothing of the size (sites x states) goes through memory: 4 bytes per 16 cells
// and direction are written and read, where storing every row takes 8 bytes a cell.
//
// The states are padded in front to 128 J (J exact: 128 (J - 1) < K <= 128 J, so
// only row 0 holds padding, kept at 0). Sums follow a fixed tree: padded state
// 128 j + 4 l + c belongs to lane l and component c; each (l, c) adds its j in
// increasing order, then (c0 + c1) + (c2 + c3), then the lanes pairwise at
// distances 16, 8, 4, 2, 1. Every fused multiply-add is an explicit one where the
// reference's compiled arithmetic has one (build with --fmad=false).
#include <algorithm>
#include <type_traits>

#include "internal.h"

namespace gp {

namespace {

constexpr int kMaxChainsPerCta = 4;  // chains per CTA: 1, 2 or 4 (the autotuner's choice)
constexpr int kChainThreads = 64;
static_assert(32 % kRowSites == 0, "kept rows at the starts of equal parts of a 32-site block");

// Arguments of the chains and blocks of a launch.
struct ChainArgs {
  int count;                          // haplotypes
  const int32_t* __restrict__ poly;
  const int32_t* __restrict__ npoly;
  const int32_t* __restrict__ nstates;
  const uint32_t* __restrict__ hvar;
  const float4* __restrict__ em;
  const float2* __restrict__ tr;
  const uint8_t* __restrict__ fl;
  const int64_t* __restrict__ row_off;  // [n] first kept row (floats): forward rows of the blocks, then backward rows
  float* __restrict__ rows;
  float* __restrict__ fac;              // [2][n][32 WB] (1 - t) / sum into every site, forward and backward
  int n, L, WB, Kp;
  float* __restrict__ hp;
  const int32_t* __restrict__ order;    // [count] haplotype of each chain pair (longest first), or null for the identity
};

// ---------------------------------------------------------------------------
// k_impute_chain: 64 threads per chain; thread `tid` owns the padded states
// 128 j + 2 tid and + 1 of every row j as a packed pair. A chain is bound by the
// latency of a site (division, state loop, sum) with one to two warps per
// scheduler, and a full batch by its instructions: four warps of half the rows
// measured the same for one haplotype (K = 1,000: 209 against 213 ns a site) and
// more for a batch (K = 400, 256 haplotypes: 439 against 358), as every warp
// repeats the division and the sum. The threads' sums meet in shared memory behind
// the site's only barrier, where every lane adds the eight partial sums of its
// group (components and distances 16 and 8) from two 16-byte loads, so that three
// shuffles finish the sum. Records and Hvar words are loaded a block ahead.
// ---------------------------------------------------------------------------

// Partial sums of the threads: lane l's pair p (components 2p, 2p + 1) at
// 12 (l & 7) + 4 (l >> 4) + 2 p + (l >> 3 & 1): the eight values of l & 7 are two
// aligned 16-byte vectors, whose halves add as packed pairs, and neither the
// stores nor the loads conflict.
constexpr int kRedStride = 12;

struct ChainSmem {
  float red[2][8 * kRedStride];
  // per block of 32 sites: emission of allele 0 and 1, t / K and 1 - t into this site; a record
  // past either end of a block is read and not used
  float4 rec[1 + 4 * 32 + 1];
};

// SOLO: one chain per CTA (its barrier is the CTA's), else a named barrier per chain.
template <int J, bool FWD, bool SOLO>
__device__ __forceinline__ void run_chain(const ChainArgs& A, ChainSmem& S, int t, int tid, int bar_id) {
  constexpr int Ks = 128 * J;
  const int np = A.npoly[t];
  const int K = A.nstates[t];
  if (np == 0 || K == 0) return;
  const int lane = tid & 31, wi = tid >> 5;
  const int kb = 2 * tid - (Ks - K);  // state of this thread's first element in row 0
  const f2 exists0 = f2_pack(kb >= 0 ? 1.f : 0.f, kb >= -1 ? 1.f : 0.f);
  const int nrow = (np + kRowSites - 1) / kRowSites;
  float* rows = A.rows + A.row_off[t] + (FWD ? 0 : (size_t)nrow * Ks) + 2 * tid;
  float* fac = A.fac + ((size_t)(FWD ? 0 : A.n) + t) * 32 * A.WB;
  const uint32_t* hv = A.hvar + (size_t)t * A.WB * A.Kp + kb;
  const float4* E = A.em + (size_t)t * A.L;
  const float2* T = A.tr + (size_t)t * A.L;
  const uint8_t* F = A.fl + (size_t)t * A.L;
  constexpr int dir = FWD ? 1 : -1;
  auto barrier = [&]() {
    if (SOLO) __syncthreads();
    else asm volatile("bar.sync %0, %1;" ::"r"(bar_id), "r"(kChainThreads) : "memory");
  };

  // Records of a block, loaded a block ahead by the first warp; Hvar words likewise, each thread its own.
  float4 pe = make_float4(0.f, 0.f, 0.f, 0.f);
  auto load_recs = [&](int b) {
    const int l = (b << 5) + lane;
    if (wi != 0 || l >= np) return;
    const float4 e = E[l];
    const bool f = F[l] != 0;  // flat and low-quality sites: emissions (1, 1), an exact factor
    const float2 tt = FWD ? (l > 0 ? T[l - 1] : make_float2(0.f, 0.f)) : T[l];
    pe = make_float4(f ? 1.0f : e.x, f ? 1.0f : e.y, tt.x, tt.y);
  };
  uint32_t w[2 * J], wn[2 * J];
  auto load_words = [&](int b) {
    const uint32_t* r = hv + (size_t)b * A.Kp;
#pragma unroll
    for (int j = 0; j < J; ++j) {
      wn[2 * j] = j > 0 || kb >= 0 ? r[128 * j] : 0u;
      wn[2 * j + 1] = j > 0 || kb >= -1 ? r[128 * j + 1] : 0u;
    }
  };

  const int b_first = FWD ? 0 : (np - 1) >> 5;
  const int b_last = FWD ? (np - 1) >> 5 : 0;
  load_recs(b_first);
  if (wi == 0) S.rec[1 + (b_first & 3) * 32 + lane] = pe;
  load_words(b_first);
  f2 x[J];  // alpha (forward) or Beta (backward)
#pragma unroll
  for (int j = 0; j < J; ++j) x[j] = f2_pack(0.f, 0.f);
  float acc = 1.f;  // AlphaSum / betaSum of the previous step
  barrier();
  const int l_first = FWD ? 0 : np - 1;
  float* const rout = &S.red[0][kRedStride * ((tid >> 1) & 7) + 4 * (tid >> 5) + 2 * (tid & 1) + ((tid >> 4) & 1)];
  const ulonglong2* const rin = reinterpret_cast<const ulonglong2*>(&S.red[0][kRedStride * (lane & 7)]);
  int parity = 0;
  float keep = 0.f;  // lane i: the factor of the block's site i
  int i = l_first & 31;
  uint32_t m = 1u << i;
  const float4* rp = nullptr;
  float4 rec = make_float4(1.f, 1.f, 0.f, 0.f);

  // Site i of the block; INIT: the first one of the chain, whose pre-emission value is 1/K.
  auto step = [&](auto init_tag) {
    constexpr bool INIT = decltype(init_tag)::value;
    const float fact1 = INIT ? 1.0f / (float)K : rec.z;
    const float fact2 = INIT ? 0.f : rec.w / acc;
    const f2 f1 = f2_pack(fact1, fact1), f2v = f2_pack(fact2, fact2);
    const float ex = rec.x, ey = rec.y;
    if (lane == i) keep = fact2;
    f2 q = f2_pack(0.f, 0.f);
#pragma unroll
    for (int j = 0; j < J; ++j) {
      const bool b0 = (w[2 * j] & m) != 0u, b1 = (w[2 * j + 1] & m) != 0u;
      f2 nx = f2_mul(f2_fma(x[j], f2v, f1), f2_pack(b0 ? ey : ex, b1 ? ey : ex));
      if (j == 0) nx = f2_mul(nx, exists0);  // padding is multiplied by 0, states by 1 (exact)
      q = j == 0 ? nx : f2_add(q, nx);
      x[j] = nx;
    }
    float v0, v1;
    f2_unpack(q, v0, v1);
    rout[parity] = __fadd_rn(v0, v1);
    i += dir;
    m = FWD ? m << 1 : m >> 1;
    rp += dir;
    rec = *rp;
    barrier();
    const ulonglong2 a = rin[parity >> 2], c = rin[(parity >> 2) + 1];
    f2_unpack(f2_add(f2_add(a.x, a.y), f2_add(c.x, c.y)), v0, v1);
    float v = __fadd_rn(v0, v1);
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, o));
    // AlphaSum = 1 at a flat first site, betaSum = 1 at a flat last site (imputation_hmm.cpp:156,285)
    acc = INIT && F[l_first] != 0 ? 1.0f : v;
    parity ^= 8 * kRedStride;
  };

  for (int b = b_first;; b += dir) {
    // the block's records and words are in place; request the next block's
#pragma unroll
    for (int j = 0; j < 2 * J; ++j) w[j] = wn[j];
    rp = &S.rec[1 + (b & 3) * 32 + i];
    rec = *rp;
    if (b != b_last) {
      load_recs(b + dir);
      load_words(b + dir);
    }
    if (b == b_first) step(std::integral_constant<bool, true>());
    const int end = FWD ? min(np - (b << 5), 32) : -1;  // i after the block
    while (i != end) {
      const int part = i / kRowSites;
      if (FWD ? i == part * kRowSites : i == (part + 1) * kRowSites - 1) {
        // the row entering this part of the block
        float* r = rows + (size_t)(b * (32 / kRowSites) + part) * Ks;
#pragma unroll
        for (int j = 0; j < J; ++j) {
          float o0, o1;
          f2_unpack(x[j], o0, o1);
          *reinterpret_cast<float2*>(r + 128 * j) = make_float2(o0, o1);
        }
      }
      const int stop = FWD ? min(end, (part + 1) * kRowSites) : part * kRowSites - 1;
      while (i != stop) step(std::integral_constant<bool, false>());
    }
    if (wi == 0) fac[(b << 5) + lane] = keep;
    if (b == b_last) break;
    if (wi == 0) S.rec[1 + ((b + dir) & 3) * 32 + lane] = pe;
    i = FWD ? 0 : 31;
    m = FWD ? 1u : 1u << 31;
    barrier();
  }
}

// Chain c = blockIdx.x * (chains per CTA) + slot is run by the 64 threads of its
// slot: haplotype order[c / 2] (c / 2 without an order), forward for even chains
// and backward for odd ones. Both warps of a chain take the same branches, so the
// chain's barrier always sees all 64 threads.
template <int J, bool SOLO>
__global__ void __launch_bounds__(SOLO ? kChainThreads : kChainThreads * kMaxChainsPerCta, 1)
    k_impute_chain(ChainArgs A) {
  __shared__ ChainSmem S[SOLO ? 1 : kMaxChainsPerCta];
  const int slot = SOLO ? 0 : threadIdx.x / kChainThreads, tid = threadIdx.x % kChainThreads;
  const int chain = SOLO ? blockIdx.x : blockIdx.x * (int)(blockDim.x / kChainThreads) + slot;
  if (chain >= 2 * A.count) return;
  const int t = A.order ? A.order[chain >> 1] : chain >> 1;
  if ((chain & 1) == 0) run_chain<J, true, SOLO>(A, S[slot], t, tid, 1 + slot);
  else run_chain<J, false, SOLO>(A, S[slot], t, tid, 1 + slot);
}

// ---------------------------------------------------------------------------
// k_impute_block: posteriors, block by block of kRowSites sites, 128 threads. Thread
// tid = 4 l + c takes its padded states 128 j + tid two rows j at a time, as a packed
// pair (rows -1 and 0 first when J is odd): the forward steps, whose values stay in
// registers, then the backward steps, the products added to the thread's two sums
// per site (one per allele). All site data is uniform and comes from shared memory;
// the loop over rows needs no communication. One lane tree per site and allele ends
// a block. Bound by issue, about 14 instructions per (site, state); to keep it so, a
// CTA takes several consecutive blocks and loads the next pair of rows and the next
// block's site data while it works on the current ones.
//
// CK, for the checkpointed modes: the same with 256 threads, thread tid taking the
// states 256 j + tid, without padding (only the last pair has absent states), and the
// sums of those modes: lanes at distances 16 .. 1, then warps at 1, 2, 4. It takes the
// blocks of one window (blockIdx.z: in which half).
// ---------------------------------------------------------------------------
constexpr int RS = kRowSites;

struct WindowArgs {
  int bf16, windows, win;  // see ckpt_layout
};

template <bool CK>
struct BlockSmem {
  // site data of two blocks
  float4 fwd[2][RS];  // t / K twice, (1 - t) / sum twice, into the site from the left
  float4 bwd[2][RS];  // the same from the right
  float2 em[2][RS];   // emissions of allele 0 and 1
  float part[2][CK ? 8 : 32][2 * RS + 4];  // [lane l (CK: warp)][value 2 site + allele]
};

// Shared-memory loads that stay where they are: moved out of the loop over rows,
// as plain loads of the same addresses would be, they do not fit the registers.
__device__ __forceinline__ void lds(unsigned addr, f2& a, f2& b) {
  asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "r"(addr));
}
__device__ __forceinline__ void lds(unsigned addr, float& a, float& b) {
  asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(a), "=f"(b) : "r"(addr));
}

// A pair of rows over the block. MASK: forward values of states that do not exist are
// held at 0 by a factor (1 elsewhere, exact). LAST: the haplotype's last block, where the site
// `last` starts the backward recursion and its posterior uses alpha alone
// (imputation_hmm.cpp:268-300).
template <bool MASK, bool LAST>
__device__ __forceinline__ void block_pair(unsigned fwd, unsigned bwd, unsigned em, uint32_t w0, uint32_t w1, f2 x,
                                           f2 y, f2 exists, int last, float (&q0)[RS], float (&q1)[RS]) {
  f2 alpha[RS];
#pragma unroll
  for (int i = 0; i < RS; ++i) {
    f2 f1, fac;
    float ea, eb;
    lds(fwd + 16 * i, f1, fac);
    lds(em + 8 * i, ea, eb);
    x = f2_mul(f2_fma(x, fac, f1), f2_pack((w0 >> i) & 1u ? eb : ea, (w1 >> i) & 1u ? eb : ea));
    if (MASK) x = f2_mul(x, exists);
    alpha[i] = x;
  }
  // the same words as new values: tests kept from the loop above would take registers
  asm volatile("" : "+r"(w0), "+r"(w1));
#pragma unroll
  for (int i = RS - 1; i >= 0; --i) {
    f2 f1, fac;
    float ea, eb;
    lds(bwd + 16 * i, f1, fac);
    lds(em + 8 * i, ea, eb);
    const bool b0 = (w0 >> i) & 1u, b1 = (w1 >> i) & 1u;
    const f2 pc = f2_fma(y, fac, f1);
    const f2 d = LAST && i == last ? alpha[i] : f2_mul(alpha[i], pc);
    y = f2_mul(pc, f2_pack(b0 ? eb : ea, b1 ? eb : ea));
    float d0, d1;
    f2_unpack(d, d0, d1);
    if (b0) q1[i] = __fadd_rn(q1[i], d0);
    else q0[i] = __fadd_rn(q0[i], d0);
    if (b1) q1[i] = __fadd_rn(q1[i], d1);
    else q0[i] = __fadd_rn(q0[i], d1);
  }
}

template <bool CK>
__global__ void __launch_bounds__(CK ? 256 : 128, CK ? 2 : 4) k_impute_block(ChainArgs A, int blocks_per,
                                                                                   WindowArgs W) {
  constexpr int NT = CK ? 256 : 128;  // threads, states of a row
  __shared__ BlockSmem<CK> S;
  const int t = A.order ? A.order[blockIdx.y] : blockIdx.y;
  const int np = A.npoly[t], K = A.nstates[t];
  const int nrow = (np + RS - 1) / RS;
  int b = blockIdx.x * blocks_per, rend = nrow;
  int64_t row0 = 0;  // CK: offset of forward row 0
  int to_bwd = 0;    // rows from a forward row to the backward one
  if constexpr (CK) {
    const CkptLayout lay = ckpt_layout(np, K, W.bf16, W.windows);
    const int half = blockIdx.z;
    int lo, hi;
    ckpt_window(lay, half, W.win, lo, hi);
    b += lo * (32 / RS);
    rend = min(nrow, hi * (32 / RS));
    // the window's rows of its chain; the other direction's beside them or among the checkpoints
    const int chain = (int)(ckpt_window_rows(lay, half, W.win) / lay.Ks) - lo * (32 / RS);
    const int other = W.bf16 ? chain + (half ? lay.wlen1 : lay.wlen0) * (32 / RS) : 0;
    row0 = (int64_t)(half == 0 ? chain : other) * lay.Ks + lay.Ks - K;
    to_bwd = half == 0 ? other - chain : chain - other;
  }
  const int bend = min(rend, b + blocks_per);
  if (b >= bend || K == 0) return;
  const int J = (K + NT - 1) >> (CK ? 8 : 7), Ks = CK ? (K + 127) & ~127 : 128 * J;
  const int pad = CK ? 0 : Ks - K;  // in front of row 0
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const float* base = A.rows + A.row_off[t] + (CK ? row0 : 0);
  const uint32_t* hvt = A.hvar + (size_t)t * A.WB * A.Kp - pad;

  // Rows j and j + 1 of this thread in block b: words and the kept values entering from both
  // sides. A state that does not exist takes those of the nearest one, so that its backward
  // values are a state's: from 0, with allele 0 everywhere, they would grow by up to 1 / min_gl
  // at each site that all states mismatch, and 0 * inf would enter the sums.
  struct Pair {
    uint32_t w0, w1;
    float a0, a1, b0, b1;
  };
  auto load = [&](int b, int j) {
    Pair p;
    const int o = NT * j + tid;
    const int o0 = CK ? min(o, K - 1) : max(o, pad), o1 = CK ? min(o + NT, K - 1) : max(o + NT, pad);
    const uint32_t* hv = hvt + (size_t)((b * RS) >> 5) * A.Kp;
    const float* ar = base + (size_t)b * Ks;
    const float* br = ar + (int64_t)(CK ? to_bwd : nrow) * Ks;
    const bool left = b > 0, right = b < nrow - 1;
    p.w0 = hv[o0];
    p.w1 = hv[o1];
    p.a0 = left ? ar[o0] : 0.f;
    p.a1 = left ? ar[o1] : 0.f;
    p.b0 = right ? br[o0] : 0.f;
    p.b1 = right ? br[o1] : 0.f;
    return p;
  };
  // Site data of a block, one site per thread of the first RS, and the site of this lane's output.
  const float2* T = A.tr + (size_t)t * A.L;
  const float* fac = A.fac + (size_t)t * 32 * A.WB;
  const float init = 1.0f / (float)K;
  float4 f = make_float4(0.f, 0.f, 0.f, 0.f), g = f;
  float2 em = make_float2(0.f, 0.f);
  int site = 0, next_site = 0;
  auto load_sites = [&](int b) {
    const int lo = b * RS + (lane >> 1);
    if (lo < np) next_site = A.poly[(size_t)t * A.L + lo];
    if (tid >= RS) return;
    const int l = b * RS + tid;
    // past the last site: the identity step
    f = g = make_float4(0.f, 0.f, 1.f, 1.f);
    em = make_float2(1.f, 1.f);
    if (l < np) {
      const float fa = fac[l], fb = fac[(size_t)A.n * 32 * A.WB + l];
      const float ta = l > 0 ? T[l - 1].x : init, tb = l < np - 1 ? T[l].x : init;
      f = make_float4(ta, ta, fa, fa);
      g = make_float4(tb, tb, fb, fb);
      const float4 ee = A.em[(size_t)t * A.L + l];
      if (A.fl[(size_t)t * A.L + l] == 0) em = make_float2(ee.x, ee.y);
    }
  };
  auto put_sites = [&](int par) {
    if (tid >= RS) return;
    S.fwd[par][tid] = f;
    S.bwd[par][tid] = g;
    S.em[par][tid] = em;
  };
  const int j0 = CK ? 0 : -(J & 1);
  const int jm = CK ? (J - 1) & ~1 : j0;  // the pair with absent states
  const f2 exists = CK ? f2_pack(NT * jm + tid < K ? 1.f : 0.f, NT * (jm + 1) + tid < K ? 1.f : 0.f)
                       : f2_pack(j0 == 0 && tid >= pad ? 1.f : 0.f, j0 == 0 || tid >= pad ? 1.f : 0.f);
  Pair n = load(b, j0);
  load_sites(b);
  put_sites(0);
  __syncthreads();
  const unsigned fwd0 = static_cast<unsigned>(__cvta_generic_to_shared(&S.fwd[0][0]));
  const unsigned bwd0 = static_cast<unsigned>(__cvta_generic_to_shared(&S.bwd[0][0]));
  const unsigned em0 = static_cast<unsigned>(__cvta_generic_to_shared(&S.em[0][0]));
  int par = 0;
#pragma unroll 1
  for (; b < bend; ++b) {
    site = next_site;
    if (b + 1 < bend) load_sites(b + 1);
    const unsigned fwd = fwd0 + par * sizeof(S.fwd[0]), bwd = bwd0 + par * sizeof(S.bwd[0]);
    const unsigned ems = em0 + par * sizeof(S.em[0]);
    const int shift = (b * RS) & 31, last = np - 1 - b * RS;
    float q0[RS], q1[RS];
#pragma unroll
    for (int i = 0; i < RS; ++i) q0[i] = q1[i] = 0.f;
    const bool final_block = b == nrow - 1;
#pragma unroll 1
    for (int j = j0; j < J; j += 2) {
      const Pair p = n;
      if (j + 2 < J) n = load(b, j + 2);
      else if (b + 1 < bend) n = load(b + 1, j0);
      const f2 x = f2_pack(p.a0, p.a1), y = f2_pack(p.b0, p.b1);
      const uint32_t w0 = p.w0 >> shift, w1 = p.w1 >> shift;
      if (final_block) block_pair<true, true>(fwd, bwd, ems, w0, w1, x, y, j == jm ? exists : f2_pack(1.f, 1.f), last, q0, q1);
      else if (j == jm) block_pair<true, false>(fwd, bwd, ems, w0, w1, x, y, exists, -1, q0, q1);
      else block_pair<false, false>(fwd, bwd, ems, w0, w1, x, y, 0, -1, q0, q1);
    }
    if constexpr (CK) {
      // reduce-scatter over lane distances 16 .. 1: value 2 site + allele ends at lane 2 site + allele
      float q[2 * RS];
#pragma unroll
      for (int i = 0; i < RS; ++i) {
        q[2 * i] = q0[i];
        q[2 * i + 1] = q1[i];
      }
#pragma unroll
      for (int h = 16; h > 0; h >>= 1) {
        const bool up = lane & h;
#pragma unroll
        for (int i = 0; i < h; ++i) {
          const float send = up ? q[i] : q[i + h], keep = up ? q[i + h] : q[i];
          q[i] = __fadd_rn(keep, __shfl_xor_sync(0xffffffffu, send, h));
        }
      }
      S.part[par][warp][lane] = q[0];
    } else {
      // Components of a lane l = tid / 4: reduce-scatter over thread distances 1 and 2.
      const int c = tid & 3;
      const bool up1 = c & 1, up2 = c & 2;
#pragma unroll
      for (int i = 0; i < RS / 2; ++i) {
        const float s0 = up1 ? q0[i] : q0[i + RS / 2], k0 = up1 ? q0[i + RS / 2] : q0[i];
        const float s1 = up1 ? q1[i] : q1[i + RS / 2], k1 = up1 ? q1[i + RS / 2] : q1[i];
        q0[i] = __fadd_rn(k0, __shfl_xor_sync(0xffffffffu, s0, 1));
        q1[i] = __fadd_rn(k1, __shfl_xor_sync(0xffffffffu, s1, 1));
      }
#pragma unroll
      for (int i = 0; i < RS / 4; ++i) {
        const float s0 = up2 ? q0[i] : q0[i + RS / 4], k0 = up2 ? q0[i + RS / 4] : q0[i];
        const float s1 = up2 ? q1[i] : q1[i + RS / 4], k1 = up2 ? q1[i + RS / 4] : q1[i];
        const int st = RS / 2 * (c & 1) + RS / 4 * (c >> 1) + i;
        const float v0 = __fadd_rn(k0, __shfl_xor_sync(0xffffffffu, s0, 2));
        const float v1 = __fadd_rn(k1, __shfl_xor_sync(0xffffffffu, s1, 2));
        *reinterpret_cast<float2*>(&S.part[par][tid >> 2][2 * st]) = make_float2(v0, v1);
      }
    }
    if (b + 1 < bend) put_sites(par ^ 1);
    __syncthreads();
    if (warp == (b & (NT / 32 - 1))) {  // the 2 RS = 32 sums of the block, the warps in turn
      float v[8];
      if constexpr (CK) {
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = S.part[par][i][lane];
#pragma unroll
        for (int h = 1; h < 8; h <<= 1)
#pragma unroll
          for (int i = 0; i < 8; i += 2 * h) v[i] = __fadd_rn(v[i], v[i + h]);
      } else {
#pragma unroll
        for (int i = 0; i < 8; ++i)
          v[i] = __fadd_rn(__fadd_rn(S.part[par][i][lane], S.part[par][i + 16][lane]),
                           __fadd_rn(S.part[par][i + 8][lane], S.part[par][i + 24][lane]));
#pragma unroll
        for (int h = 4; h > 0; h >>= 1)
#pragma unroll
          for (int i = 0; i < h; ++i) v[i] = __fadd_rn(v[i], v[i + h]);
      }
      // prob_hid of the two alleles; k_impute_finish turns them into HP
      if ((lane >> 1) <= last) A.hp[(size_t)t * 2 * A.L + 2 * site + (lane & 1)] = v[0];
    }
    par ^= 1;
  }
}

}  // namespace

// Rows of 128 states for K states (the J of launch_impute_chain).
int impute_groups(int K) { return std::max(1, (K + 127) / 128); }

static int chain_args(ImputeWork& w, float* hp, int first, int count, ChainArgs& a) {
  if (count < 0) count = w.n;
  if (first < 0 || first + count > w.n || (first > 0 && !w.order.ptr)) return GP_E_ARG;
  a.count = count;
  a.poly = w.poly.as<int32_t>();
  a.npoly = w.npoly.as<int32_t>();
  a.nstates = w.nstates.as<int32_t>();
  a.hvar = w.hvar.as<uint32_t>();
  a.em = w.em.as<float4>();
  a.tr = w.tr.as<float2>();
  a.fl = w.fl.as<uint8_t>();
  a.row_off = w.row_off.as<int64_t>();
  a.rows = w.rows.as<float>();
  a.fac = w.fac.as<float>();
  a.n = w.n;
  a.L = w.L;
  a.WB = w.WB;
  a.Kp = w.Kp;
  a.hp = hp;
  a.order = w.order.ptr ? w.order.as<int32_t>() + first : nullptr;
  return GP_OK;
}

int launch_impute_chain(int J, ImputeWork& w, cudaStream_t s, int first, int count, int cpc) {
  ChainArgs a;
  if (chain_args(w, nullptr, first, count, a) != GP_OK || cpc < 1 || cpc > kMaxChainsPerCta) return GP_E_ARG;
  if (a.count == 0) return GP_OK;
  const int g = (2 * a.count + cpc - 1) / cpc, threads = kChainThreads * cpc;
#define GP_CHAIN(JJ)                                           \
  case JJ:                                                     \
    if (cpc == 1) k_impute_chain<JJ, true><<<g, threads, 0, s>>>(a);  \
    else k_impute_chain<JJ, false><<<g, threads, 0, s>>>(a);   \
    return GP_OK;
  switch (J) {
    GP_CHAIN(1) GP_CHAIN(2) GP_CHAIN(3) GP_CHAIN(4) GP_CHAIN(5) GP_CHAIN(6) GP_CHAIN(7) GP_CHAIN(8)
    GP_CHAIN(9) GP_CHAIN(10) GP_CHAIN(11) GP_CHAIN(12) GP_CHAIN(13) GP_CHAIN(14) GP_CHAIN(15) GP_CHAIN(16)
    default: return GP_E_ARG;
  }
#undef GP_CHAIN
}

static_assert(2 * kRowSites == 32, "k_impute_block: one lane per sum of a block");

// Blocks per CTA: enough to hide the loads of each, while some eight CTAs per SM are left.
static int blocks_per_cta(long long total) { return (int)std::max(1ll, std::min(16ll, total / (8 * 148))); }

int launch_impute_block(int max_poly, ImputeWork& w, float* hp, cudaStream_t s, int first, int count) {
  ChainArgs a;
  if (chain_args(w, hp, first, count, a) != GP_OK) return GP_E_ARG;
  const int blocks = (max_poly + kRowSites - 1) / kRowSites;
  if (a.count == 0 || blocks == 0) return GP_OK;
  const int per = blocks_per_cta((long long)blocks * a.count);
  k_impute_block<false><<<dim3((blocks + per - 1) / per, a.count), 128, 0, s>>>(a, per, {});
  return GP_OK;
}

int launch_ckpt_posteriors(bool bf16, int windows, int win, int wlen, ImputeWork& w, float* hp, cudaStream_t s,
                           int first, int count) {
  ChainArgs a;
  if (chain_args(w, hp, first, count, a) != GP_OK) return GP_E_ARG;
  const int blocks = wlen * (32 / kRowSites);
  if (a.count == 0 || blocks == 0) return GP_OK;
  const int per = blocks_per_cta(2ll * blocks * a.count);
  k_impute_block<true><<<dim3((blocks + per - 1) / per, a.count, 2), 256, 0, s>>>(a, per, {bf16, windows, win});
  return GP_OK;
}

}  // namespace gp

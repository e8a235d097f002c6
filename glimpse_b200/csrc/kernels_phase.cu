// The 8-hypothesis phasing HMM with Gibbs phase resampling
// (phase/src/models/phasing_hmm.{h,cpp}, rephaseHaplotypes :247-302).
//
// Four kernels after the VAR list: k_phase_chain (the two sequential passes of
// every target, side by side), k_phase_units (what combines a forward and a
// backward message, all units in parallel), k_phase_draw (the diplotype chain)
// and the write-back. Messages are stored in global memory as [row][k][8].
#include <cub/block/block_scan.cuh>

#include "internal.h"
#include "phase.h"

namespace gp {

namespace {

constexpr int NW = 8;  // virtual warps, see the order of the sums

// ---------------------------------------------------------------------------
// VAR list and segmentation (phasing_hmm.cpp:65-140)
// ---------------------------------------------------------------------------
template <int THREADS, int ITEMS>
__global__ void k_build_vars(const int32_t* __restrict__ poly, const int32_t* __restrict__ npoly,
                             const uint8_t* __restrict__ h0, const uint8_t* __restrict__ h1,
                             const uint8_t* __restrict__ flat, const uint8_t* __restrict__ lq, int L,
                             const int32_t* __restrict__ tsel, PhaseVars V) {
  typedef cub::BlockScan<int, THREADS> Scan;
  __shared__ typename Scan::TempStorage tmp;
  __shared__ int carry[3];
  const int b = blockIdx.x;
  const int t = tsel ? tsel[b] : b;
  const int np = npoly[t];
  const int32_t* pl = poly + (size_t)t * L;
  const uint8_t* H0 = h0 + (size_t)t * L;
  const uint8_t* H1 = h1 + (size_t)t * L;
  const uint8_t* FL = flat + (size_t)t * L;
  int32_t* vrel = V.rel + (size_t)b * V.lv;
  uint8_t* vcode = V.code + (size_t)b * V.lv;
  int32_t* vseg = V.seg + (size_t)b * V.lv;
  int32_t* vmiss = V.miss + (size_t)b * V.lv;
  int32_t* mrel = V.miss_rel + (size_t)b * V.lv;
  int32_t* sstart = V.seg_start + (size_t)b * (V.lv + 2);
  if (threadIdx.x < 3) carry[threadIdx.x] = 0;
  __syncthreads();
  for (int base = 0; base < np; base += THREADS * ITEMS) {
    int isv[ITEMS], isph[ITEMS], isfh[ITEMS], code[ITEMS];
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
      const int l = base + threadIdx.x * ITEMS + i;
      isv[i] = isph[i] = isfh[i] = 0;
      code[i] = 0;
      if (l < np) {
        const int s = pl[l];
        const int a0 = H0[s], a1 = H1[s];
        const bool nf = !FL[s] && !lq[s];
        if (nf) {
          isv[i] = 1;
          if (a0 != a1) { isph[i] = 1; code[i] = 0; }
          else code[i] = VT_HOM | (a0 << 3);
        } else if (a0 != a1) {
          isv[i] = 1;
          isfh[i] = 1;
          code[i] = VT_FLAT | (a0 << 3);
        }
      }
    }
    int exv[ITEMS], exh[ITEMS], exm[ITEMS];
    int tv, th, tm;
    Scan(tmp).ExclusiveSum(isv, exv, tv);
    __syncthreads();
    Scan(tmp).ExclusiveSum(isph, exh, th);
    __syncthreads();
    Scan(tmp).ExclusiveSum(isfh, exm, tm);
    const int cv = carry[0], ch = carry[1], cmm = carry[2];
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
      const int l = base + threadIdx.x * ITEMS + i;
      if (l < np && isv[i]) {
        const int vi = cv + exv[i];
        const int hc = ch + exh[i];  // peak hets before this entry
        int c = code[i];
        int seg;
        if (isph[i]) {
          c = hc % 3;  // VAR_TYP = n_het % 3
          seg = hc / 3;
          if (hc > 0 && hc % 3 == 0) sstart[seg] = vi;
        } else {
          seg = (hc > 0 ? hc - 1 : 0) / 3;
        }
        vrel[vi] = l;
        vcode[vi] = (uint8_t)c;
        vseg[vi] = seg;
        vmiss[vi] = isfh[i] ? cmm + exm[i] : -1;
        if (isfh[i]) mrel[cmm + exm[i]] = l;
      }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      carry[0] = cv + tv;
      carry[1] = ch + th;
      carry[2] = cmm + tm;
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    const int nv = carry[0], nh = carry[1], nm = carry[2];
    const int nseg = (nh > 0 ? nh - 1 : 0) / 3 + 1;
    sstart[0] = 0;
    sstart[nseg] = nv;
    V.nvar[b] = nv;
    V.nseg[b] = nseg;
    V.nmiss[b] = nm;
  }
}

// Per-entry transitions (conditioning_set.h:101-105, as getTransition is called
// in phasing_hmm.cpp:152,201 and phasing_hmm.h:381) and segment flags.
__device__ __forceinline__ float transition(const double* __restrict__ cm, int prev, int next, const ModelConst& mc);

__global__ void k_var_records(const int32_t* __restrict__ tsel, const int32_t* __restrict__ poly, int L,
                              const double* __restrict__ cm, ModelConst mc, PhaseVars V) {
  const int b = blockIdx.y;
  const int t = tsel ? tsel[b] : b;
  const int nv = V.nvar[b];
  const int32_t* pl = poly + (size_t)t * L;
  const int32_t* vrel = V.rel + (size_t)b * V.lv;
  const int32_t* vseg = V.seg + (size_t)b * V.lv;
  const int32_t* sstart = V.seg_start + (size_t)b * (V.lv + 2);
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nv; i += gridDim.x * blockDim.x) {
    const int s = pl[vrel[i]];
    float yn = 0.f;
    if (i + 1 < nv) yn = transition(cm, s, pl[vrel[i + 1]], mc);
    V.yt_next[(size_t)b * V.lv + i] = yn;
    float yp = 0.f;
    if (i > 0) yp = transition(cm, pl[vrel[i - 1]], s, mc);
    V.yt_prev[(size_t)b * V.lv + i] = yp;
    const int seg = vseg[i];
    const int locus = i - sstart[seg];
    const int seglen = sstart[seg + 1] - sstart[seg];
    const int fl = (locus == 0 ? 1 : 0) | (locus == seglen - 1 ? 2 : 0);
    V.flags[(size_t)b * V.lv + i] = (uint8_t)fl;
    const int x = vrel[i] | ((int)V.code[(size_t)b * V.lv + i] << 24) | (fl << 28);
    const int miss = V.miss[(size_t)b * V.lv + i];
    V.recb[(size_t)b * V.lv + i] = make_int4(x, seg, miss, __float_as_int(yn));
    V.recf[(size_t)b * V.lv + i] = make_int4(x, seg, miss, __float_as_int(yp));
  }
}

// ---------------------------------------------------------------------------
// The order of the sums over states
//
// Every sum over the K states (probSumH at each VAR site, the transition sums
// of TRANS_HAP and the flat-het sums) has one fixed tree, so that the draws it
// feeds do not depend on the launch shape: state k belongs to lane k % 32 of
// virtual warp (k / 32) % 8; each (virtual warp, lane) adds its states in
// increasing order, the lanes of a virtual warp are added pairwise at distances
// 16, 8, 4, 2, 1, and the virtual warps pairwise at distances 1, 2, 4.
// ---------------------------------------------------------------------------
constexpr unsigned kFull = 0xffffffffu;

__device__ __forceinline__ float shfl_x(float v, int o) { return __shfl_xor_sync(kFull, v, o); }
__device__ __forceinline__ f2 shfl_x(f2 v, int o) {
  float lo, hi;
  f2_unpack(v, lo, hi);
  return f2_pack(shfl_x(lo, o), shfl_x(hi, o));
}

// horizontal_add of 8 lanes as the reference's AVX reduction orders it
// (phasing_hmm.h:47-57): ((v0+v4)+(v1+v5)) + ((v2+v6)+(v3+v7)).
__device__ __forceinline__ float hadd8(const float (&v)[8]) {
  const float l0 = __fadd_rn(v[0], v[4]), l1 = __fadd_rn(v[1], v[5]);
  const float l2 = __fadd_rn(v[2], v[6]), l3 = __fadd_rn(v[3], v[7]);
  return __fadd_rn(__fadd_rn(l0, l1), __fadd_rn(l2, l3));
}
// The same over packed pairs (v0,v1) (v2,v3) (v4,v5) (v6,v7). The value does
// not change when the hypotheses are permuted by h -> h ^ f (additions commute).
__device__ __forceinline__ float hadd8(const f2 (&v)[4]) {
  float l0, l1, l2, l3;
  f2_unpack(f2_add(v[0], v[2]), l0, l1);
  f2_unpack(f2_add(v[1], v[3]), l2, l3);
  return __fadd_rn(__fadd_rn(l0, l1), __fadd_rn(l2, l3));
}

// Hypothesis allele at a het of type `typ` (ALLELE(HAP_NUMBER-h-1, 2-typ), phasing_hmm.h:45).
__device__ __forceinline__ int hyp_allele(int h, int typ) { return ((7 - h) >> (2 - typ)) & 1; }

__device__ __forceinline__ float transition(const double* __restrict__ cm, int prev, int next, const ModelConst& mc) {
  const double d = mc.nrho * (cm[next] - cm[prev]);
  double x = -expm1(d);
  x = x < 1e-7 ? 1e-7 : (x > mc.one_l ? mc.one_l : x);
  return (float)x;  // conditioning_set.h:101-105
}

// ---------------------------------------------------------------------------
// k_phase_chain: the sequential part of the phasing HMM. One CTA runs one chain,
// the backward (phasing_hmm.cpp:193-245) or the forward pass (:142-191) of one
// diploid target; neither needs the other, since everything that combines the
// two (TRANS_HAP, IMPUTE_FLAT_HET, the diplotype draws) reads messages that both
// store: the backward pass at segment starts, the forward pass at segment ends,
// both at flat hets.
//
// A chain is bound by the latency of one VAR site: totals -> two divisions ->
// the state loop -> the sums over states -> totals, with about one warp per
// scheduler, so every instruction of a site counts. The shape follows from that:
//  - Four warps of V = 2 virtual warps each (two of V = 4 where many chains share an
//    SM, Context::run_phase); a thread holds the 8 hypothesis messages of its V J
//    states in registers, as packed pairs. J is exact: a launch holds the targets
//    with 256 (J - 1) < K <= 256 J, so only the last V slots can be empty and the
//    state loop is one straight-line block.
//  - Register slot s of lane `lane` holds hypothesis s ^ f, f a function of the
//    lane: the reduce-scatter over the lanes then always keeps its lower slots
//    and sends its upper ones, with no selects. The virtual warps are held in
//    lane-swapped order too, so the first levels scatter them and 17 (V = 2) or 33
//    (V = 4) shuffles reduce 16 or 32 values.
//  - The warps' sums meet in shared memory behind the site's only barrier, in
//    four copies (one per f % 4), so that every lane reads all 8 totals in its
//    own slot order with 16-byte loads from one 128-byte row per warp.
//  - Emissions need no table: at a peak hom the mismatching states are multiplied
//    by ed / ee and the others left alone (a factor of 1); at a peak het of type
//    typ a slot's factor depends on the state allele, slot bit 2 - typ and a lane
//    constant, so two values a state serve all slots.
//  - Hets, the start and segment starts change the messages or the factors in
//    place before one common loop: variants of the loop, joined by the compiler
//    with register moves, cost a quarter of the instructions.
// Measured, whole phasing per iteration: 11 targets of a 2,503 x 30,011 panel at
// K 130-900 28.1 -> 8.0 ms; 256 targets of a 10,000 x 150,000 panel at K 400-1,200
// 116 -> 46 ms (both passes in one 256-thread CTA before). 243 warp instructions a
// site at J = 2, 313 at J = 4; two warps of one virtual warp each instead of one of two: slower
// at 11 targets (16.1 against 14.2 ms, first version) and at 256.
// ---------------------------------------------------------------------------
// V virtual warps per warp: 8 / V warps, 256 / V threads a chain.
template <int V>
struct ChainShared {
  float4 red[2][8 / V][4][2];  // [buffer][warp][copy][slots 0-3 / 4-7]
  int4 rec[128];            // ring of four chunks of 32 records
  float* rows;     // the chain's stored messages: segments, then flat hets
  float* segsum;   // their sums and totals
  float* segtot;
  float* misssum;
  int nseg;
};

__device__ __forceinline__ f2 lo2(float4 v) { return f2_pack(v.x, v.y); }
__device__ __forceinline__ f2 hi2(float4 v) { return f2_pack(v.z, v.w); }

// Set s of a lane's registers holds virtual warp V * warp + (s ^ set_swap), slot s
// hypothesis s ^ lane_class.
template <int V>
__device__ __forceinline__ int set_swap(int lane) { return V == 2 ? lane >> 4 : lane >> 3; }
template <int V>
__device__ __forceinline__ int lane_class(int lane) { return V == 2 ? (lane >> 1) & 7 : lane & 7; }
// The copy of the sums that a lane writes: the four lanes of a class write all four.
template <int V>
__device__ __forceinline__ int lane_copy(int lane) { return V == 2 ? (lane & 1) | ((lane >> 4) << 1) : lane >> 3; }

// A warp's sums of its virtual warps over the lanes, added: hypothesis lane_class,
// the same in the four lanes of that class.
template <int V>
__device__ __forceinline__ float warp_scatter(const f2 (&part)[V][4]) {
  f2 v[4];
  float x, y;
  if constexpr (V == 2) {
#pragma unroll
    for (int q = 0; q < 4; ++q) v[q] = f2_add(part[0][q], shfl_x(part[1][q], 16));
    v[0] = f2_add(v[0], shfl_x(v[2], 8));
    v[1] = f2_add(v[1], shfl_x(v[3], 8));
    v[0] = f2_add(v[0], shfl_x(v[1], 4));
    f2_unpack(v[0], x, y);
    x = __fadd_rn(x, shfl_x(y, 2));
    x = __fadd_rn(x, shfl_x(x, 1));
    return __fadd_rn(x, shfl_x(x, 16));
  } else {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      v[q] = f2_add(part[0][q], shfl_x(part[2][q], 16));
      const f2 u = f2_add(part[1][q], shfl_x(part[3][q], 16));
      v[q] = f2_add(v[q], shfl_x(u, 8));
    }
    v[0] = f2_add(v[0], shfl_x(v[2], 4));
    v[1] = f2_add(v[1], shfl_x(v[3], 4));
    v[0] = f2_add(v[0], shfl_x(v[1], 2));
    f2_unpack(v[0], x, y);
    x = __fadd_rn(x, shfl_x(y, 1));
    x = __fadd_rn(x, shfl_x(x, 8));
    return __fadd_rn(x, shfl_x(x, 16));
  }
}

// The totals over the warps, tot[q] = slots (2q, 2q + 1) of a lane of class f.
template <int CW>
__device__ __forceinline__ void read_totals(const float4 (*red)[4][2], int f, f2 (&tot)[4]) {
  f2 t[CW][4];
#pragma unroll
  for (int w = 0; w < CW; ++w) {
    const float4* r = red[w][f & 3];
    const float4 a = r[f >> 2], b = r[(f >> 2) ^ 1];
    t[w][0] = lo2(a);
    t[w][1] = hi2(a);
    t[w][2] = lo2(b);
    t[w][3] = hi2(b);
  }
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    tot[q] = f2_add(t[0][q], t[1][q]);
    if (CW == 4) tot[q] = f2_add(tot[q], f2_add(t[CW - 2][q], t[CW - 1][q]));
  }
}

__device__ __forceinline__ void cp_async4(void* smem, const void* gmem) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(
                   static_cast<unsigned>(__cvta_generic_to_shared(smem))), "l"(gmem));
}
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(
                   static_cast<unsigned>(__cvta_generic_to_shared(smem))), "l"(gmem));
}
__device__ __forceinline__ void cp_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// Fields of a packed VAR record's x (PhaseVars::recb / recf).
constexpr uint32_t kRecFlat = (uint32_t)VT_FLAT << 24, kRecAlt = 1u << 27, kRecFirst = 1u << 28, kRecLast = 1u << 29;

// The update of a peak het of type TYP, prob = (prob * ntp + tF) * emission
// (phasing_hmm.h:140-366). A state allele that differs from `flip` (which
// carries the lane's hypothesis bit) emits ee in the slots whose bit 2 - TYP is 0.
template <int NS, int TYP>
__device__ __forceinline__ void het_update(f2 (&prob)[NS][4], const uint32_t (&w)[NS], uint32_t m, uint32_t flip,
                                           float ee, float ed, const f2 (&tF)[4], f2 ntp) {
#pragma unroll
  for (int i = 0; i < NS; ++i) {
    const bool hit = ((w[i] & m) ^ flip) != 0u;
    const float x = hit ? ee : ed, y = hit ? ed : ee;
    const f2 xx = f2_pack(x, x), yy = f2_pack(y, y), xy = f2_pack(x, y);
#pragma unroll
    for (int q = 0; q < 4; ++q)
      prob[i][q] = f2_mul(f2_fma(prob[i][q], ntp, tF[q]), TYP == 2 ? xy : (TYP == 1 ? (q & 1) : (q >> 1)) ? yy : xx);
  }
}

template <int J, int V>
__global__ void __launch_bounds__(256 / V, phase_chains_per_sm(J, V == 4))
    k_phase_chain(const int32_t* __restrict__ tsel, const int32_t* __restrict__ nstates,
                  const int32_t* __restrict__ npoly, const uint32_t* __restrict__ hvar, int WB, int Kp, PhaseVars P,
                  PhaseStore S, ModelConst mc) {
  constexpr int NS = V * J, CW = 8 / V, CT = 32 * CW;
  __shared__ ChainShared<V> sm;
  __shared__ uint32_t words[2][NS][CT];  // Hvar words of two 32-site blocks, each thread's own
  const int b = S.order[blockIdx.x >> 1];
  const bool fwd = blockIdx.x & 1;
  const int t = tsel ? tsel[b] : b;
  const int K = nstates[t];
  const int nv = P.nvar[b];
  if (nv == 0) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int f = lane_class<V>(lane), copy = lane_copy<V>(lane);
  const uint32_t* hv = hvar + (size_t)t * WB * Kp;
  const int nblk_poly = (npoly[t] + 31) >> 5;
  const int4* recs = (fwd ? P.recf : P.recb) + (size_t)b * P.lv;
  // slot i = V j + s: state k = 256 j + kb[s]. A slot without a state (of the last V)
  // repeats the last state, words and all, and does not count in the sums: its messages
  // are those of a state. (As a state of its own, with allele 0 everywhere, it would grow by
  // ee / ed at every hom that all real states mismatch, and overflow.)
  int kb[V], kw[V];
  bool last[V];
  f2 exists[V];
#pragma unroll
  for (int s = 0; s < V; ++s) {
    kb[s] = 32 * (V * warp + (s ^ set_swap<V>(lane))) + lane;
    last[s] = 256 * (J - 1) + kb[s] < K;
    kw[s] = min(256 * (J - 1) + kb[s], K - 1);
    exists[s] = last[s] ? f2_pack(1.f, 1.f) : f2_pack(0.f, 0.f);
  }
  auto has = [&](int i) { return i < NS - V || last[i % V]; };

  f2 prob[NS][4];
  uint32_t w[NS];
  f2 tot[4];
  float sumT;

  auto fetch_words = [&](int blk) {
    if (blk < 0 || blk >= nblk_poly) return;
#pragma unroll
    for (int i = 0; i < NS; ++i)
      cp_async4(&words[blk & 1][i][tid],
                hv + (size_t)blk * Kp + (i < NS - V ? 256 * (i / V) + kb[i % V] : kw[i % V]));
  };
  auto read_words = [&](int blk) {
#pragma unroll
    for (int i = 0; i < NS; ++i) w[i] = words[blk & 1][i][tid];
  };
  // Rows in slot order, only the halves back in place; k_phase_units undoes the rest of h -> h ^ f.
  auto store_rows = [&](float* dst) {
#pragma unroll
    for (int i = 0; i < NS; ++i) {
      if (!has(i)) continue;
      float v[8];
#pragma unroll
      for (int q = 0; q < 4; ++q) f2_unpack(prob[i][q], v[2 * q], v[2 * q + 1]);
      float4* d4 = reinterpret_cast<float4*>(dst + (size_t)(256 * (i / V) + kb[i % V]) * 8);
      d4[f >> 2] = make_float4(v[0], v[1], v[2], v[3]);
      d4[(f >> 2) ^ 1] = make_float4(v[4], v[5], v[6], v[7]);
    }
  };
  auto store_sums = [&](float* dst) {  // thread 0 holds the totals in natural order (f = 0)
    float4* d4 = reinterpret_cast<float4*>(dst);
    float v[8];
#pragma unroll
    for (int q = 0; q < 4; ++q) f2_unpack(tot[q], v[2 * q], v[2 * q + 1]);
    d4[0] = make_float4(v[0], v[1], v[2], v[3]);
    d4[1] = make_float4(v[4], v[5], v[6], v[7]);
  };
  // records of steps s = 0 .. nv-1 (entry s forward, nv-1-s backward)
  auto fetch_recs = [&](int c) {
    const int s = (c << 5) + lane;
    if (s < nv) cp_async16(&sm.rec[s & 127], recs + (fwd ? s : nv - 1 - s));
  };
  if (warp == 0) {
    fetch_recs(0);
    fetch_recs(1);
  }
  if (tid == 0) {
    // pool: backward rows of the segments and of the flat hets, then the forward rows of both
    const int nseg = P.nseg[b];
    const int64_t so = S.seg_off[b] + (fwd ? S.seg_total : 0), mo = S.miss_off[b] + (fwd ? S.miss_total : 0);
    sm.nseg = nseg;
    sm.rows = S.pool + S.pool_off[b] + (fwd ? (size_t)(nseg + P.nmiss[b]) * K * 8 : 0);
    sm.segsum = S.seg_sum + so * 8;
    sm.segtot = S.seg_tot + so;
    sm.misssum = S.miss_sum + mo * 8;
  }
  cp_wait_all();
  __syncthreads();
  uint32_t rx;
  float yt;
  auto read_rec = [&](int s) {
    const int4 r = sm.rec[s & 127];
    rx = (uint32_t)r.x;
    yt = __int_as_float(r.w);
  };
  read_rec(0);
  const int dir = fwd ? 1 : -1;
  int cur = (int)(rx & 0xffffffu) >> 5, nxt = cur + dir;
  fetch_words(cur);
  cp_wait_all();
  read_words(cur);
  fetch_words(nxt);
  const float Kf = (float)K;
  const float mism = mc.ed_phs / mc.ee_phs;
  const uint32_t collapse = fwd ? kRecFirst : kRecLast;           // first entry of a segment in sweep direction
  const uint32_t keep = (fwd ? kRecLast : kRecFirst) | kRecFlat;  // entries whose messages are stored
  int buf = 0;
  float* const rbase = reinterpret_cast<float*>(&sm.red[0][warp][copy]) + ((f & 4) | ((f & 3) ^ copy));

  // Stores the messages of step s, whose record's x is cx.
  auto keep_messages = [&](int s, uint32_t cx) {
    const int4 rr = sm.rec[s & 127];
    if ((cx & keep & ~kRecFlat) && !(fwd && s == nv - 1)) {
      store_rows(sm.rows + (size_t)rr.y * K * 8);
      if (tid == 0) {
        store_sums(sm.segsum + (size_t)rr.y * 8);
        sm.segtot[rr.y] = sumT;
      }
    }
    if (cx & kRecFlat) {
      store_rows(sm.rows + (size_t)(sm.nseg + rr.z) * K * 8);
      if (tid == 0) store_sums(sm.misssum + (size_t)rr.z * 8);
    }
  };

  int s = 0;
  if (rx & kRecFlat) {
    // INIT at a flat het: every message is 1 / (8 K) (phasing_hmm.h:140-366)
    const float v = 1.0f / (float)(8u * (unsigned)K);
#pragma unroll
    for (int i = 0; i < NS; ++i)
#pragma unroll
      for (int q = 0; q < 4; ++q) prob[i][q] = f2_pack(v, v);
#pragma unroll
    for (int q = 0; q < 4; ++q) tot[q] = f2_pack(0.125f, 0.125f);
    sumT = 1.0f;
    keep_messages(0, rx);
    s = 1;
    read_rec(1);  // unused when there is no such step
  } else {
    // INIT elsewhere is the emission alone: (0 * x + 1 * (K / (K * 1))) * emission
#pragma unroll
    for (int i = 0; i < NS; ++i)
#pragma unroll
      for (int q = 0; q < 4; ++q) prob[i][q] = f2_pack(0.f, 0.f);
#pragma unroll
    for (int q = 0; q < 4; ++q) tot[q] = f2_pack(1.f, 1.f);
    sumT = 1.0f;
    yt = Kf;
  }
  while (s < nv) {
    // Chunk c of 32 steps: chunk c + 1 has landed and chunk c + 2 goes to the ring
    // slots of chunk c - 2, which no warp reads any more.
    const int c = s >> 5;
    if (warp == 0) {
      cp_wait_all();
      fetch_recs(c + 2);
    }
    __syncthreads();
    const int send = min(nv, (c + 1) << 5);
    for (; s < send; ++s) {
      const int blk = (int)(rx & 0xffffffu) >> 5;
      if (blk != cur) {
        cp_wait_all();
        if (blk != nxt) {
          fetch_words(blk);
          cp_wait_all();
        }
        read_words(blk);
        cur = blk;
        nxt = blk + dir;
        fetch_words(nxt);
      }
      const uint32_t m = 1u << (rx & 31);
      const uint32_t typ = (rx >> 24) & 7u;
      const float sc = yt / __fmul_rn(Kf, sumT);
      const float np = (1.0f - yt) / sumT;
      const f2 scp = f2_pack(sc, sc);
      f2 ntp = f2_pack(np, np);
      f2 tF[4], part[V][4];
#pragma unroll
      for (int q = 0; q < 4; ++q) tF[q] = f2_mul(tot[q], scp);
      if (rx & collapse) {  // COLLAPSE: every message of a state becomes their sum (SUMK)
#pragma unroll
        for (int i = 0; i < NS; ++i) {
          const float k = hadd8(prob[i]);
#pragma unroll
          for (int q = 0; q < 4; ++q) prob[i][q] = f2_pack(k, k);
        }
      }
      if (typ < 3u) {
        // A peak het updates in place; the loop below then leaves the messages as they are.
        const uint32_t flip = ((f >> (2 - typ)) & 1) ? m : 0u;
        if (typ == 0) het_update<NS, 0>(prob, w, m, flip, mc.ee_phs, mc.ed_phs, tF, ntp);
        else if (typ == 1) het_update<NS, 1>(prob, w, m, flip, mc.ee_phs, mc.ed_phs, tF, ntp);
        else het_update<NS, 2>(prob, w, m, flip, mc.ee_phs, mc.ed_phs, tF, ntp);
#pragma unroll
        for (int q = 0; q < 4; ++q) tF[q] = f2_pack(0.f, 0.f);
        ntp = f2_pack(1.f, 1.f);
      }
      const float fac = typ == VT_HOM ? mism : 1.0f;
      const uint32_t flip = (rx & kRecAlt) ? m : 0u;
#pragma unroll
      for (int i = 0; i < NS; ++i) {
        const float x = ((w[i] & m) ^ flip) != 0u ? fac : 1.0f;
        const f2 xx = f2_pack(x, x);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          prob[i][q] = f2_mul(f2_fma(prob[i][q], ntp, tF[q]), xx);
          // the last V slots count by a factor of exactly 1 or 0
          if (i < V) part[i][q] = i < NS - V ? prob[i][q] : f2_mul(prob[i][q], exists[i]);
          else part[i % V][q] = i < NS - V ? f2_add(part[i % V][q], prob[i][q])
                                           : f2_fma(prob[i][q], exists[i % V], part[i % V][q]);
        }
      }
      rbase[buf * (CW * 32)] = warp_scatter<V>(part);
      const uint32_t cx = rx;
      read_rec(s + 1);
      __syncthreads();
      read_totals<CW>(sm.red[buf], f, tot);
      sumT = hadd8(tot);
      buf ^= 1;
      if (cx & keep) keep_messages(s, cx);
    }
  }
  cp_wait_all();
}

// ---------------------------------------------------------------------------
// k_phase_units: the sums that combine a forward and a backward message. Unit
// u < nseg - 1 of an entry is the boundary between segments u and u + 1 (TRANS_HAP,
// phasing_hmm.h:376-397): the 8 x 8 transition sums and, for every diplotype the
// chain could arrive with, the diplotype that SAMPLE_DIP (:400-411) draws next. The
// others are its flat hets (IMPUTE_FLAT_HET, :414-447). Units are independent; the
// work is reading two stored messages (64 bytes a state and unit) and 64 (or 16)
// multiply-adds a state.
//
// A CTA of 8 warps (a virtual warp each) takes every gridDim.x-th unit of one entry.
// Thread tid owns the states tid + 256 j; the values of the next steps (a step: one j
// of a unit) are always in flight, copied by cp.async into slots that only its warp
// reads, also while a unit is summed up, so that memory does not idle. Messages stay in the
// chain's slot order (h -> h ^ f within the halves, f & 3 of the lane); the sums over
// the lanes go through shared memory, where writing a value to the row of its
// hypothesis pair undoes the permutation at no cost, 16 rows at a time; two lanes
// add a row's 32 values in the fixed tree. One barrier a unit; a unit's last steps
// and draws fall to one warp, the next unit's to the next warp.
// ---------------------------------------------------------------------------
constexpr int kUnitStages = 4;
constexpr int kUnitsPerCta = 8;  // at least, where an entry has that many

struct UnitSmem {
  float4 row[kUnitStages][4][256];     // two messages of a thread's state
  uint32_t word[kUnitStages][256];     // its Hvar word (flat hets)
  float tr[NW][16][36];                // values of 16 hypothesis pairs by lane (lanes 2i + p at 16 p + i)
  float red[2][NW][64];                // the warps' sums
  float hp[64];
  float sc[2][16];                     // a unit's factors
};

__device__ __forceinline__ float warps_sum(const float (*red)[64], int i) {
  const float a = __fadd_rn(red[0][i], red[1][i]), b = __fadd_rn(red[2][i], red[3][i]);
  const float c = __fadd_rn(red[4][i], red[5][i]), d = __fadd_rn(red[6][i], red[7][i]);
  return __fadd_rn(__fadd_rn(a, b), __fadd_rn(c, d));
}

// The sums over the lanes of the 16 rows that the warp wrote to tr: row lane / 2,
// valid in both lanes of a pair.
__device__ __forceinline__ float rows_sum(const float (*tr)[36], int lane) {
  const ulonglong2* r = reinterpret_cast<const ulonglong2*>(&tr[lane >> 1][16 * (lane & 1)]);
  const ulonglong2 v0 = r[0], v1 = r[1], v2 = r[2], v3 = r[3];  // lanes 2i + p, i = 0-3, 4-7, 8-11, 12-15
  const f2 a = f2_add(f2_add(v0.x, v2.x), f2_add(v1.x, v3.x));  // distances 16 and 8
  const f2 b = f2_add(f2_add(v0.y, v2.y), f2_add(v1.y, v3.y));
  float x, y;
  f2_unpack(f2_add(a, b), x, y);                                // distance 4
  x = __fadd_rn(x, y);                                          // distance 2
  return __fadd_rn(x, shfl_x(x, 1));
}

__global__ void __launch_bounds__(256, 2) k_phase_units(const int32_t* __restrict__ tsel,
                                                        const int32_t* __restrict__ nstates,
                                                        const uint32_t* __restrict__ hvar, int WB, int Kp, PhaseVars P,
                                                        PhaseStore S, uint64_t seed, int iteration,
                                                        const int32_t* __restrict__ target_ids,
                                                        uint32_t narrow) {
  extern __shared__ __align__(16) char smem_raw[];
  UnitSmem& sm = *reinterpret_cast<UnitSmem*>(smem_raw);
  const int b = S.order[blockIdx.y];
  const int t = tsel ? tsel[b] : b;
  const int K = nstates[t];
  const int nv = P.nvar[b];
  const int nseg = P.nseg[b], nmiss = P.nmiss[b];
  const int nb = nv > 0 ? nseg - 1 : 0;  // boundaries
  const int nu = nb + nmiss;
  if ((int)blockIdx.x >= nu) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nj = (K + 255) >> 8;
  // the chain's slot s of a half holds hypothesis s ^ f
  const int f = ((narrow >> nj) & 1u ? lane_class<4>(lane) : lane_class<2>(lane)) & 3;
  const float* pool = S.pool + S.pool_off[b];
  const size_t rowf = (size_t)K * 8, fbase = (size_t)(nseg + nmiss) * rowf;
  const int64_t so = S.seg_off[b], mo = S.miss_off[b];
  const int32_t* mrel = P.miss_rel + (size_t)b * P.lv;
  const uint32_t rng_target = target_ids ? (uint32_t)target_ids[b] : (uint32_t)t;

  // Steps in flight. A warp's states are 1 KB of either row, copied in whole 512-byte
  // pieces: lane l takes the 16-byte chunks l and l + 32, half l & 1 of state l >> 1 (+ 16).
  int iu = blockIdx.x, ij = 0, istage = 0;
  const int kl = 32 * warp + (lane >> 1);
  const uint32_t* hv = hvar + (size_t)t * WB * Kp + tid;
  const float *px = pool, *py = pool;
  const uint32_t* pw = nullptr;  // Hvar words of the unit's site, null at boundaries
  auto site_of = [&](int u) { return u >= nb && u < nu ? mrel[u - nb] : 0; };
  int site = site_of(iu);  // of the unit begun next
  auto begin_unit = [&]() {
    if (iu >= nu) return;
    // boundary u: forward row at the end of segment u, backward row at the start of u + 1;
    // flat het m: backward and forward row
    const bool flat = iu >= nb;
    px = (flat ? pool + (size_t)(nseg + iu - nb) * rowf : pool + fbase + (size_t)iu * rowf) + 256 * warp + 4 * lane;
    py = flat ? px + fbase : pool + (size_t)(iu + 1) * rowf + 256 * warp + 4 * lane;
    pw = flat ? hv + (size_t)(site >> 5) * Kp : nullptr;
    site = site_of(iu + gridDim.x);
  };
  auto issue = [&]() {
    if (iu < nu) {
      const int k = kl + 256 * ij;
      float4* d = &sm.row[istage][lane & 1][kl];
      if (k < K) {
        cp_async16(d, px);
        cp_async16(d + 512, py);
      }
      if (k + 16 < K) {
        cp_async16(d + 16, px + 128);
        cp_async16(d + 528, py + 128);
      }
      if (pw && tid + 256 * ij < K) cp_async4(&sm.word[istage][tid], pw + 256 * ij);
      px += 2048;
      py += 2048;
    }
    asm volatile("cp.async.commit_group;\n" ::);
    istage = istage + 1 == kUnitStages ? 0 : istage + 1;
    if (++ij == nj) {
      ij = 0;
      iu += gridDim.x;
      begin_unit();
    }
  };
  begin_unit();
  // A unit's factors, one per thread of the first 16. Boundary: fact1 of hypothesis h (8 of them) and fact2;
  // flat het: the reciprocal sums of the backward and the forward message.
  float s0 = 0.f, s1 = 1.f, s2 = 0.f;
  auto load_factors = [&](int u) {
    if (tid >= 16 || u >= nu) return;
    if (u < nb) {
      s0 = S.seg_sum[(S.seg_total + so + u) * 8 + (tid & 7)];
      s1 = S.seg_tot[S.seg_total + so + u];
      s2 = P.yt_next[(size_t)b * P.lv + P.seg_start[(size_t)b * (P.lv + 2) + u + 1] - 1];
    } else {
      s0 = S.miss_sum[((tid < 8 ? 0 : S.miss_total) + mo + u - nb) * 8 + (tid & 7)];
    }
  };
  auto put_factors = [&](int u, int par) {
    if (tid >= 16 || u >= nu) return;
    float v;
    if (u >= nb) v = 1.0f / s0;
    else if (tid < 8) v = __fmul_rn(s0 / s1, s2) / (float)K;
    else v = (1.0f - s2) / s1;
    sm.sc[par][tid] = v;
  };
#pragma unroll
  for (int i = 0; i < kUnitStages - 1; ++i) issue();
  load_factors(blockIdx.x);
  put_factors(blockIdx.x, 0);
  __syncthreads();
  // where this lane writes value (s1, s2) (low two bits each) of 16 pairs: row (s1 ^ f) * 4 + (s2 ^ f)
  float* const trp = &sm.tr[warp][0][16 * (lane & 1) + (lane >> 1)];
  const int fx = 5 * f;
  int cstage = 0, par = 0, owner = 0;
  for (int u = blockIdx.x; u < nu; u += gridDim.x) {
    load_factors(u + gridDim.x);
    if (u < nb) {
      const float4* c4 = reinterpret_cast<const float4*>(sm.sc[par]);
      float fact1[8];
#pragma unroll
      for (int h = 0; h < 8; ++h) fact1[h] = sm.sc[par][(h & 4) | ((h & 3) ^ f)];
      const float fact2 = c4[2].x;
      f2 acc[8][4];
#pragma unroll
      for (int h = 0; h < 8; ++h)
#pragma unroll
        for (int q = 0; q < 4; ++q) acc[h][q] = f2_pack(0.f, 0.f);
      for (int j = 0; j < nj; ++j) {
        asm volatile("cp.async.wait_group %0;\n" ::"n"(kUnitStages - 2) : "memory");
        __syncwarp();  // the other lanes' pieces have landed, and the slot issued next is no longer read
        if (tid + 256 * j < K) {
          const float4 x0 = sm.row[cstage][0][tid], x1 = sm.row[cstage][1][tid];
          const float4 y0 = sm.row[cstage][2][tid], y1 = sm.row[cstage][3][tid];
          const float p[8] = {x0.x, x0.y, x0.z, x0.w, x1.x, x1.y, x1.z, x1.w};
          const f2 n[4] = {lo2(y0), hi2(y0), lo2(y1), hi2(y1)};
#pragma unroll
          for (int h = 0; h < 8; ++h) {
            const float p0 = fmaf(p[h], fact2, fact1[h]);
            const f2 pp = f2_pack(p0, p0);
#pragma unroll
            for (int q = 0; q < 4; ++q) acc[h][q] = f2_fma(pp, n[q], acc[h][q]);
          }
        }
        issue();
        cstage = cstage + 1 == kUnitStages ? 0 : cstage + 1;
      }
#pragma unroll
      for (int r = 0; r < 4; ++r) {  // rounds of 16 pairs: halves r / 2 of h1 and r % 2 of h2
#pragma unroll
        for (int i = 0; i < 16; i += 2) {
          float lo, hi;
          f2_unpack(acc[4 * (r >> 1) + (i >> 2)][2 * (r & 1) + ((i >> 1) & 1)], lo, hi);
          trp[(i ^ fx) * 36] = lo;
          trp[((i + 1) ^ fx) * 36] = hi;
        }
        __syncwarp();
        const float v = rows_sum(sm.tr[warp], lane);
        const int i = lane >> 1;
        if ((lane & 1) == 0) sm.red[par][warp][(4 * (r >> 1) + (i >> 2)) * 8 + 4 * (r & 1) + (i & 3)] = v;
        __syncwarp();
      }
      put_factors(u + gridDim.x, par ^ 1);
      __syncthreads();
      if (warp == owner) {
        sm.hp[lane] = warps_sum(sm.red[par], lane);
        sm.hp[lane + 32] = warps_sum(sm.red[par], lane + 32);
        __syncwarp();
        float sumHP = 0.f;
#pragma unroll
        for (int h1 = 0; h1 < 8; ++h1) {
          float v[8];
#pragma unroll
          for (int h2 = 0; h2 < 8; ++h2) v[h2] = sm.hp[h1 * 8 + h2];
          sumHP = __fadd_rn(sumHP, hadd8(v));
        }
        const int prev = lane & 7;
        const bool bad1 = isnan(sumHP) || isinf(sumHP) || sumHP < 1.17549435e-38f;
        float dp[8], sd = 0.f;
#pragma unroll
        for (int d = 0; d < 8; ++d) {
          dp[d] = __fmul_rn(sm.hp[prev * 8 + d] / sumHP, sm.hp[(7 - prev) * 8 + (7 - d)] / sumHP);
          sd = __fadd_rn(sd, dp[d]);
        }
        const bool bad = bad1 || isnan(sd) || isinf(sd) || sd < 1.17549435e-38f;
        const float uu = __fmul_rn(canonical_float(stream_word(seed, RNG_PHASE, iteration, rng_target,
                                                               (uint64_t)(u + 1))), sd);
        int nd = 7;
        float cs = dp[0];
#pragma unroll
        for (int d = 0; d < 7; ++d) {
          if (nd == 7 && uu <= cs) nd = d;
          cs = __fadd_rn(cs, dp[d + 1]);
        }
        if (bad) nd = prev;  // an invalid sum keeps the diplotype and raises the entry's error flag
        uint32_t mine = lane < 8 ? ((uint32_t)nd << (3 * prev)) | ((bad ? 1u : 0u) << (24 + prev)) : 0u;
        mine = __reduce_or_sync(kFull, mine);
        if (lane == 0) S.next[so + u] = mine;
      }
    } else {
      const int m = u - nb;
      const uint32_t bit = 1u << (mrel[m] & 31);
      float sR[8], sL[8], v[16];
#pragma unroll
      for (int h = 0; h < 8; ++h) {
        sR[h] = sm.sc[par][(h & 4) | ((h & 3) ^ f)];
        sL[h] = sm.sc[par][8 + ((h & 4) | ((h & 3) ^ f))];
        v[h] = v[h + 8] = 0.f;
      }
      for (int j = 0; j < nj; ++j) {
        asm volatile("cp.async.wait_group %0;\n" ::"n"(kUnitStages - 2) : "memory");
        __syncwarp();  // the other lanes' pieces have landed, and the slot issued next is no longer read
        if (tid + 256 * j < K) {
          const float4 x0 = sm.row[cstage][0][tid], x1 = sm.row[cstage][1][tid];
          const float4 y0 = sm.row[cstage][2][tid], y1 = sm.row[cstage][3][tid];
          const bool alt = (sm.word[cstage][tid] & bit) != 0u;
          const float ip[8] = {x0.x, x0.y, x0.z, x0.w, x1.x, x1.y, x1.z, x1.w};
          const float pr[8] = {y0.x, y0.y, y0.z, y0.w, y1.x, y1.y, y1.z, y1.w};
#pragma unroll
          for (int h = 0; h < 8; ++h) {
            const float p1 = __fmul_rn(ip[h], sR[h]);
            const float p2 = __fmul_rn(pr[h], sL[h]);
            if (alt) v[8 + h] = fmaf(p1, p2, v[8 + h]); else v[h] = fmaf(p1, p2, v[h]);
          }
        }
        issue();
        cstage = cstage + 1 == kUnitStages ? 0 : cstage + 1;
      }
      // rows: allele * 8 + hypothesis
#pragma unroll
      for (int i = 0; i < 16; ++i) trp[(i ^ f) * 36] = v[i];
      __syncwarp();
      const float x = rows_sum(sm.tr[warp], lane);
      if ((lane & 1) == 0) sm.red[par][warp][lane >> 1] = x;
      __syncwarp();
      put_factors(u + gridDim.x, par ^ 1);
      __syncthreads();
      if (warp == owner && lane < 8) {
        const float t0 = warps_sum(sm.red[par], lane), t1 = warps_sum(sm.red[par], lane + 8);
        const float r = t1 / __fadd_rn(t0, t1);
        S.of1[(mo + m) * 8 + lane] = fmaxf(0.0f, fminf(1.0f, r));
      }
    }
    par ^= 1;
    owner = (owner + 1) & (NW - 1);
  }
  asm volatile("cp.async.wait_all;\n" ::: "memory");
}

// The diplotype chain of one entry per warp: the first draw (phasing_hmm.cpp:249-256)
// and then the drawn successor of every boundary.
__global__ void k_phase_draw(const int32_t* __restrict__ tsel, int n, PhaseVars P, PhaseStore S, uint64_t seed,
                             int iteration, const int32_t* __restrict__ target_ids) {
  const int i = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (i >= n) return;
  const int lane = threadIdx.x & 31;
  const int b = S.order[i];
  const int t = tsel ? tsel[b] : b;
  const int nv = P.nvar[b], nseg = P.nseg[b];
  const uint32_t rng_target = target_ids ? (uint32_t)target_ids[b] : (uint32_t)t;
  const int64_t so = S.seg_off[b];
  int d0 = 7;
  uint32_t err = 0u;
  if (nv > 0) {
    const float* ps = S.seg_sum + so * 8;
    const float pt = S.seg_tot[so];
    float dp[8];
    float sd = 0.f;
    for (int d = 0; d < 8; ++d) {
      dp[d] = __fmul_rn(ps[d] / pt, ps[7 - d] / pt);
      sd = __fadd_rn(sd, dp[d]);
    }
    const float u = __fmul_rn(canonical_float(stream_word(seed, RNG_PHASE, iteration, rng_target, 0)), sd);
    float cs = dp[0];
    for (int d = 0; d < 7; ++d) {
      if (u <= cs) { d0 = d; break; }
      cs = __fadd_rn(cs, dp[d + 1]);
    }
  }
  if (lane == 0) S.dip[so] = d0;
  const int nb = nv > 0 ? nseg - 1 : 0;
  int d = d0;
  for (int base = 0; base < nb; base += 32) {
    const uint32_t mine = base + lane < nb ? S.next[so + base + lane] : 0u;
    const int c = min(32, nb - base);
    int out = 0;
    for (int j = 0; j < c; ++j) {
      const uint32_t m = __shfl_sync(kFull, mine, j);
      err |= (m >> (24 + d)) & 1u;
      d = (m >> (3 * d)) & 7;
      if (lane == j) out = d;
    }
    if (base + lane < nb) S.dip[so + base + lane + 1] = out;
  }
  if (lane == 0) S.err[b] = (int32_t)err;
}

// Allele write-back for peak and flat hets (phasing_hmm.cpp:260-292).
__global__ void k_phase_writeback(const int32_t* __restrict__ tsel, const int32_t* __restrict__ poly, int L,
                                  PhaseVars V, PhaseStore S, ModelConst mc, uint64_t seed, int iteration,
                                  const int32_t* __restrict__ target_ids, uint8_t* __restrict__ h0,
                                  uint8_t* __restrict__ h1) {
  const int b = blockIdx.y;
  const int t = tsel ? tsel[b] : b;
  const int nv = V.nvar[b];
  const int nseg = V.nseg[b];
  const uint32_t rng_target = target_ids ? (uint32_t)target_ids[b] : (uint32_t)t;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nv; i += gridDim.x * blockDim.x) {
    const int code = V.code[(size_t)b * V.lv + i];
    const int typ = code & 7;
    if (typ == VT_HOM) continue;
    const int l = V.rel[(size_t)b * V.lv + i];
    const int s = poly[(size_t)t * L + l];
    const int seg = V.seg[(size_t)b * V.lv + i];
    const int i0 = S.dip[S.seg_off[b] + seg];
    const int i1 = 7 - i0;
    if (typ < 3) {
      h0[(size_t)t * L + s] = (uint8_t)hyp_allele(i0, typ);
      h1[(size_t)t * L + s] = (uint8_t)hyp_allele(i1, typ);
    } else {
      const int m = V.miss[(size_t)b * V.lv + i];
      const float* of = S.of1 + (S.miss_off[b] + m) * 8;
      const float h0a0 = 1.0f - of[i0], h0a1 = of[i0];
      const float h1a0 = 1.0f - of[i1], h1a1 = of[i1];
      float p01 = __fmul_rn(fmaf(h0a0, mc.ee_phs, __fmul_rn(h0a1, mc.ed_phs)),
                            fmaf(h1a1, mc.ee_phs, __fmul_rn(h1a0, mc.ed_phs)));
      float p10 = __fmul_rn(fmaf(h0a1, mc.ee_phs, __fmul_rn(h0a0, mc.ed_phs)),
                            fmaf(h1a0, mc.ee_phs, __fmul_rn(h1a1, mc.ed_phs)));
      float sum = __fadd_rn(p01, p10);
      p01 = fminf(fmaxf(p01 / sum, 0.0f), 1.0f);
      p10 = fminf(fmaxf(p10 / sum, 0.0f), 1.0f);
      sum = __fadd_rn(p01, p10);
      const float u = canonical_float(stream_word(seed, RNG_PHASE, iteration, rng_target, (uint64_t)(nseg + m)));
      const bool rf = __dmul_rn((double)u, (double)sum) < (double)p01;
      h0[(size_t)t * L + s] = (uint8_t)(!rf);  // H0 written twice, H1 untouched (phasing_hmm.cpp:283-284)
    }
  }
}

// Shuffle of hets at monomorphic sites (phasing_hmm.cpp:293-301): the m-th such
// het draws word nseg + nmiss + m of the target's phasing stream.
template <int THREADS, int ITEMS>
__global__ void k_mono_shuffle(const int32_t* __restrict__ tsel, const int32_t* __restrict__ polyidx, int L,
                               PhaseVars V, uint64_t seed, int iteration, const int32_t* __restrict__ target_ids,
                               uint8_t* __restrict__ h0, uint8_t* __restrict__ h1) {
  typedef cub::BlockScan<int, THREADS> Scan;
  __shared__ typename Scan::TempStorage tmp;
  __shared__ int carry;
  const int b = blockIdx.x;
  const int t = tsel ? tsel[b] : b;
  const uint32_t rng_target = target_ids ? (uint32_t)target_ids[b] : (uint32_t)t;
  const uint64_t base_word = (uint64_t)V.nseg[b] + (uint64_t)V.nmiss[b];
  uint8_t* H0 = h0 + (size_t)t * L;
  uint8_t* H1 = h1 + (size_t)t * L;
  const int32_t* pi = polyidx + (size_t)t * L;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  for (int base = 0; base < L; base += THREADS * ITEMS) {
    int v[ITEMS], ex[ITEMS], tot;
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
      const int s = base + threadIdx.x * ITEMS + i;
      v[i] = (s < L && pi[s] < 0 && H0[s] != H1[s]) ? 1 : 0;
    }
    Scan(tmp).ExclusiveSum(v, ex, tot);
    const int c = carry;
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
      if (!v[i]) continue;
      const int s = base + threadIdx.x * ITEMS + i;
      const float u = canonical_float(stream_word(seed, RNG_PHASE, iteration, rng_target, base_word + c + ex[i]));
      const bool rf = u < 0.5f;
      H0[s] = (uint8_t)rf;
      H1[s] = (uint8_t)!rf;
    }
    __syncthreads();
    if (threadIdx.x == 0) carry = c + tot;
    __syncthreads();
  }
}

}  // namespace

void launch_build_vars(const int32_t* tsel, int nb, const int32_t* poly, const int32_t* npoly, const uint8_t* h0,
                       const uint8_t* h1, const uint8_t* flat, const uint8_t* lq, int L, PhaseVars V,
                       cudaStream_t s) {
  k_build_vars<512, 8><<<nb, 512, 0, s>>>(poly, npoly, h0, h1, flat, lq, L, tsel, V);
}

void launch_var_records(const int32_t* tsel, int nb, const int32_t* poly, int L, const double* cm,
                        const ModelConst& mc, PhaseVars V, cudaStream_t s) {
  k_var_records<<<dim3(32, nb), 256, 0, s>>>(tsel, poly, L, cm, mc, V);
}

int launch_phase_chain(int J, bool narrow, const int32_t* tsel, int nb, const int32_t* nstates, const uint32_t* hvar,
                       int WB, int Kp, const int32_t* npoly, PhaseVars P, PhaseStore S, const ModelConst& mc,
                       cudaStream_t s) {
  if (narrow && J > kPhaseNarrowJ) return GP_E_ARG;
#define GP_CHAIN(JJ, VV) \
  k_phase_chain<JJ, VV><<<2 * nb, 256 / VV, 0, s>>>(tsel, nstates, npoly, hvar, WB, Kp, P, S, mc)
  switch (J + (narrow ? 10 : 0)) {
    case 1: GP_CHAIN(1, 2); break;
    case 2: GP_CHAIN(2, 2); break;
    case 3: GP_CHAIN(3, 2); break;
    case 4: GP_CHAIN(4, 2); break;
    case 5: GP_CHAIN(5, 2); break;
    case 6: GP_CHAIN(6, 2); break;
    case 7: GP_CHAIN(7, 2); break;
    case 8: GP_CHAIN(8, 2); break;
    case 11: GP_CHAIN(1, 4); break;
    case 12: GP_CHAIN(2, 4); break;
    case 13: GP_CHAIN(3, 4); break;
    case 14: GP_CHAIN(4, 4); break;
    case 15: GP_CHAIN(5, 4); break;
    default: return GP_E_ARG;
  }
#undef GP_CHAIN
  return GP_OK;
}

int launch_phase_units(int max_units, uint32_t narrow, const int32_t* tsel, int nb, const int32_t* nstates,
                       const uint32_t* hvar, int WB, int Kp, PhaseVars P, PhaseStore S, uint64_t seed, int iteration,
                       const int32_t* target_ids, cudaStream_t s) {
  if (max_units > 0) {
    if (set_smem_limit_once<k_phase_units>((int)sizeof(UnitSmem)) != cudaSuccess) return GP_E_CUDA;
    const int g = (max_units + kUnitsPerCta - 1) / kUnitsPerCta;
    k_phase_units<<<dim3(g, nb), 256, sizeof(UnitSmem), s>>>(tsel, nstates, hvar, WB, Kp, P, S, seed, iteration,
                                                             target_ids, narrow);
  }
  return GP_OK;
}

void launch_phase_draw(const int32_t* tsel, int nb, PhaseVars P, PhaseStore S, uint64_t seed, int iteration,
                       const int32_t* target_ids, cudaStream_t s) {
  k_phase_draw<<<(nb + 3) / 4, 128, 0, s>>>(tsel, nb, P, S, seed, iteration, target_ids);
}

void launch_phase_writeback(const int32_t* tsel, int nb, const int32_t* poly, const int32_t* polyidx, int L,
                            PhaseVars V, PhaseStore S, const ModelConst& mc, uint64_t seed, int iteration,
                            const int32_t* target_ids, uint8_t* h0, uint8_t* h1, cudaStream_t s) {
  dim3 g(64, nb);
  k_phase_writeback<<<g, 256, 0, s>>>(tsel, poly, L, V, S, mc, seed, iteration, target_ids, h0, h1);
  k_mono_shuffle<512, 8><<<nb, 512, 0, s>>>(tsel, polyidx, L, V, seed, iteration, target_ids, h0, h1);
}

}  // namespace gp

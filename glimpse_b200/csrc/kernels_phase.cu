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
//  - Four warps of two virtual warps each; a thread holds the 8 hypothesis
//    messages of its 2 J states in registers, as packed pairs. J is exact: a
//    launch holds the targets with 256 (J - 1) < K <= 256 J, so only the last
//    two slots can be empty and the state loop is one straight-line block.
//  - Register slot s of lane `lane` holds hypothesis s ^ f, f a function of the
//    lane: the reduce-scatter over the lanes then always keeps its lower slots
//    and sends its upper ones, with no selects. The upper half warp also holds
//    the two virtual warps in swapped order, so the first level scatters the
//    virtual warps and 17 shuffles reduce 16 values.
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
// 116 -> 56 ms (both passes in one 256-thread CTA before). 235 warp instructions a
// site at J = 2; two warps of one virtual warp each instead of one of two: slower
// at 11 targets (16.1 against 14.2 ms, first version) and at 256.
// ---------------------------------------------------------------------------
constexpr int CT = 128;       // threads of a chain
constexpr int CW = CT / 32;   // warps

struct ChainShared {
  float4 red[2][CW][4][2];  // [buffer][warp][copy][slots 0-3 / 4-7]
  int4 rec[128];            // ring of four chunks of 32 records
  float* rows;     // the chain's stored messages: segments, then flat hets
  float* segsum;   // their sums and totals
  float* segtot;
  float* misssum;
  int nseg;
};

__device__ __forceinline__ f2 lo2(float4 v) { return f2_pack(v.x, v.y); }
__device__ __forceinline__ f2 hi2(float4 v) { return f2_pack(v.z, v.w); }

// A warp's sums of its two virtual warps over the lanes, added: hypothesis
// lane_class(lane) of the pair, the same in the four lanes of that class.
__device__ __forceinline__ float warp_scatter(const f2 (&part)[2][4]) {
  f2 v[4];
  float x, y;
#pragma unroll
  for (int q = 0; q < 4; ++q) v[q] = f2_add(part[0][q], shfl_x(part[1][q], 16));
  v[0] = f2_add(v[0], shfl_x(v[2], 8));
  v[1] = f2_add(v[1], shfl_x(v[3], 8));
  v[0] = f2_add(v[0], shfl_x(v[1], 4));
  f2_unpack(v[0], x, y);
  x = __fadd_rn(x, shfl_x(y, 2));
  x = __fadd_rn(x, shfl_x(x, 1));
  return __fadd_rn(x, shfl_x(x, 16));
}

// The totals over the warps, tot[q] = slots (2q, 2q + 1) of a lane of class f.
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
  for (int q = 0; q < 4; ++q) tot[q] = f2_add(f2_add(t[0][q], t[1][q]), f2_add(t[2][q], t[3][q]));
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

template <int J>
__global__ void __launch_bounds__(CT, J <= 2 ? 5 : J <= 4 ? 4 : J <= 5 ? 3 : 2)
    k_phase_chain(const int32_t* __restrict__ tsel, const int32_t* __restrict__ nstates,
                  const int32_t* __restrict__ npoly, const uint32_t* __restrict__ hvar, int WB, int Kp, PhaseVars P,
                  PhaseStore S, ModelConst mc) {
  constexpr int NS = 2 * J;
  __shared__ ChainShared sm;
  __shared__ uint32_t words[2][NS][CT];  // Hvar words of two 32-site blocks, each thread's own
  const int b = S.order[blockIdx.x >> 1];
  const bool fwd = blockIdx.x & 1;
  const int t = tsel ? tsel[b] : b;
  const int K = nstates[t];
  const int nv = P.nvar[b];
  if (nv == 0) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int f = (lane >> 1) & 7;                        // slot s holds hypothesis s ^ f
  const int copy = (lane & 1) | ((lane >> 4) << 1);     // the copy of the sums that this lane writes
  const uint32_t* hv = hvar + (size_t)t * WB * Kp;
  const int nblk_poly = (npoly[t] + 31) >> 5;
  const int4* recs = (fwd ? P.recf : P.recb) + (size_t)b * P.lv;
  // slot (j, s): state k = 256 j + kb[s]; the virtual warps swapped in the upper half warp
  int kb[2];
  bool last[2];
  f2 exists[2];
#pragma unroll
  for (int s = 0; s < 2; ++s) {
    kb[s] = 32 * (2 * warp + (s ^ (lane >> 4))) + lane;
    last[s] = 256 * (J - 1) + kb[s] < K;
    exists[s] = last[s] ? f2_pack(1.f, 1.f) : f2_pack(0.f, 0.f);
  }
  auto has = [&](int i) { return i < 2 * J - 2 || last[i & 1]; };

  f2 prob[NS][4];
  uint32_t w[NS];
  f2 tot[4];
  float sumT;

  auto fetch_words = [&](int blk) {
    if (blk < 0 || blk >= nblk_poly) return;
#pragma unroll
    for (int i = 0; i < NS; ++i)
      if (has(i)) cp_async4(&words[blk & 1][i][tid], hv + (size_t)blk * Kp + 256 * (i >> 1) + kb[i & 1]);
  };
  auto read_words = [&](int blk) {
#pragma unroll
    for (int i = 0; i < NS; ++i) w[i] = has(i) ? words[blk & 1][i][tid] : 0u;
  };
  // Rows in slot order, only the halves back in place; k_phase_units undoes the rest of h -> h ^ f.
  auto store_rows = [&](float* dst) {
#pragma unroll
    for (int i = 0; i < NS; ++i) {
      if (!has(i)) continue;
      float v[8];
#pragma unroll
      for (int q = 0; q < 4; ++q) f2_unpack(prob[i][q], v[2 * q], v[2 * q + 1]);
      float4* d4 = reinterpret_cast<float4*>(dst + (size_t)(256 * (i >> 1) + kb[i & 1]) * 8);
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
      f2 tF[4], part[2][4];
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
          // the last two slots count by a factor of exactly 1 or 0
          if (i < 2) part[i][q] = i < NS - 2 ? prob[i][q] : f2_mul(prob[i][q], exists[i]);
          else part[i & 1][q] = i < NS - 2 ? f2_add(part[i & 1][q], prob[i][q])
                                           : f2_fma(prob[i][q], exists[i & 1], part[i & 1][q]);
        }
      }
      rbase[buf * (CW * 32)] = warp_scatter(part);
      const uint32_t cx = rx;
      read_rec(s + 1);
      __syncthreads();
      read_totals(sm.red[buf], f, tot);
      sumT = hadd8(tot);
      buf ^= 1;
      if (cx & keep) keep_messages(s, cx);
    }
  }
  cp_wait_all();
}

// ---------------------------------------------------------------------------
// k_phase_units: the sums that combine a forward and a backward message, one CTA
// of 8 warps (a virtual warp each) per unit. Unit u < nseg - 1 of an entry is the
// boundary between segments u and u + 1 (TRANS_HAP, phasing_hmm.h:376-397): the 8 x 8
// transition sums and, for every diplotype the chain could arrive with, the
// diplotype that SAMPLE_DIP (:400-411) draws next. The others are its flat hets
// (IMPUTE_FLAT_HET, :414-447). Units are independent, so this is bound by
// reading the stored messages (64 bytes a state and unit).
// ---------------------------------------------------------------------------
// Reduce-scatter of N values over the lanes (distances 16, 8, 4, 2, 1); a lane
// keeps the upper half of the values where its bit of the distance is set, so
// lane l ends with values 2 l and 2 l + 1 of 64, or value l >> 1 of 16.
template <int N>
__device__ __forceinline__ void lane_scatter(float (&v)[N], int lane) {
  int n = N;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    if (n > 1) {
      n >>= 1;
      const bool up = lane & o;
#pragma unroll
      for (int i = 0; i < N / 2; ++i) {
        if (i >= n) break;
        const float send = up ? v[i] : v[i + n];
        const float keep = up ? v[i + n] : v[i];
        v[i] = __fadd_rn(keep, shfl_x(send, o));
      }
    } else {
      v[0] = __fadd_rn(v[0], shfl_x(v[0], o));
    }
  }
}

// A stored row of state k in natural hypothesis order: position p of a half holds
// hypothesis p ^ (f & 3) of that half, f the class of the state's lane in the chain.
__device__ __forceinline__ void load_row(const float* row, int f, float (&v)[8]) {
  const float4* r4 = reinterpret_cast<const float4*>(row);
  const float4 a = r4[0], b = r4[1];
  const bool x1 = f & 1, x2 = f & 2;
  float u[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
  for (int h = 0; h < 8; ++h) v[h] = x1 ? u[h ^ 1] : u[h];
#pragma unroll
  for (int h = 0; h < 8; ++h) u[h] = x2 ? v[h ^ 2] : v[h];
#pragma unroll
  for (int h = 0; h < 8; ++h) v[h] = u[h];
}

__device__ __forceinline__ float warps_sum(const float (*red)[64], int i) {
  const float a = __fadd_rn(red[0][i], red[1][i]), b = __fadd_rn(red[2][i], red[3][i]);
  const float c = __fadd_rn(red[4][i], red[5][i]), d = __fadd_rn(red[6][i], red[7][i]);
  return __fadd_rn(__fadd_rn(a, b), __fadd_rn(c, d));
}

__global__ void __launch_bounds__(256, 2) k_phase_units(const int32_t* __restrict__ tsel,
                                                        const int32_t* __restrict__ nstates,
                                                        const uint32_t* __restrict__ hvar, int WB, int Kp, PhaseVars P,
                                                        PhaseStore S, uint64_t seed, int iteration,
                                                        const int32_t* __restrict__ target_ids) {
  __shared__ float red[NW][64];
  __shared__ float hp[64];
  const int b = S.order[blockIdx.y];
  const int t = tsel ? tsel[b] : b;
  const int K = nstates[t];
  const int nv = P.nvar[b];
  const int nseg = P.nseg[b], nmiss = P.nmiss[b];
  const int nb = nv > 0 ? nseg - 1 : 0;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int f = (lane >> 1) & 7;
  const float* pool = S.pool + S.pool_off[b];
  const size_t fbase = (size_t)(nseg + nmiss) * K * 8;
  const uint32_t rng_target = target_ids ? (uint32_t)target_ids[b] : (uint32_t)t;
  for (int u = blockIdx.x; u < nb + nmiss; u += gridDim.x) {
    if (u < nb) {
      const int64_t so = S.seg_off[b] + u;
      const float* fsum = S.seg_sum + (S.seg_total + so) * 8;
      const float sumT = S.seg_tot[S.seg_total + so];
      const float yt = P.yt_next[(size_t)b * P.lv + P.seg_start[(size_t)b * (P.lv + 2) + u + 1] - 1];
      const float fact2 = (1.0f - yt) / sumT;
      float fact1[8];
#pragma unroll
      for (int h = 0; h < 8; ++h) fact1[h] = __fmul_rn(fsum[h] / sumT, yt) / (float)K;
      float acc[64];
#pragma unroll
      for (int i = 0; i < 64; ++i) acc[i] = 0.f;
      const float* fr = pool + fbase + (size_t)u * K * 8;
      const float* nr = pool + (size_t)(u + 1) * K * 8;
      for (int k = tid; k < K; k += 256) {
        float p[8], n[8];
        load_row(fr + (size_t)k * 8, f, p);
        load_row(nr + (size_t)k * 8, f, n);
#pragma unroll
        for (int h1 = 0; h1 < 8; ++h1) {
          const float p0 = fmaf(p[h1], fact2, fact1[h1]);
#pragma unroll
          for (int h2 = 0; h2 < 8; ++h2) acc[h1 * 8 + h2] = fmaf(p0, n[h2], acc[h1 * 8 + h2]);
        }
      }
      lane_scatter<64>(acc, lane);
      red[warp][2 * lane] = acc[0];
      red[warp][2 * lane + 1] = acc[1];
      __syncthreads();
      if (tid < 64) hp[tid] = warps_sum(red, tid);
      __syncthreads();
      if (warp == 0) {
        float sumHP = 0.f;
#pragma unroll
        for (int h1 = 0; h1 < 8; ++h1) {
          float v[8];
#pragma unroll
          for (int h2 = 0; h2 < 8; ++h2) v[h2] = hp[h1 * 8 + h2];
          sumHP = __fadd_rn(sumHP, hadd8(v));
        }
        const int prev = lane & 7;
        const bool bad1 = isnan(sumHP) || isinf(sumHP) || sumHP < 1.17549435e-38f;
        float dp[8], sd = 0.f;
#pragma unroll
        for (int d = 0; d < 8; ++d) {
          dp[d] = __fmul_rn(hp[prev * 8 + d] / sumHP, hp[(7 - prev) * 8 + (7 - d)] / sumHP);
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
        if (lane == 0) S.next[so] = mine;
      }
      __syncthreads();
    } else {
      const int m = u - nb;
      const int64_t mo = S.miss_off[b] + m;
      const float* bsum = S.miss_sum + mo * 8;
      const float* fsum = S.miss_sum + (S.miss_total + mo) * 8;
      const int l = P.miss_rel[(size_t)b * P.lv + m];
      const uint32_t* hv = hvar + ((size_t)t * WB + (l >> 5)) * Kp;
      float sR[8], sL[8], v[16];
#pragma unroll
      for (int h = 0; h < 8; ++h) {
        sR[h] = 1.0f / bsum[h];
        sL[h] = 1.0f / fsum[h];
        v[h] = v[h + 8] = 0.f;
      }
      const float* br = pool + (size_t)(nseg + m) * K * 8;
      const float* fr = br + fbase;
      for (int k = tid; k < K; k += 256) {
        const bool bit = (hv[k] >> (l & 31)) & 1u;
        float ip[8], pr[8];
        load_row(br + (size_t)k * 8, f, ip);
        load_row(fr + (size_t)k * 8, f, pr);
#pragma unroll
        for (int h = 0; h < 8; ++h) {
          const float p1 = __fmul_rn(ip[h], sR[h]);
          const float p2 = __fmul_rn(pr[h], sL[h]);
          if (bit) v[8 + h] = fmaf(p1, p2, v[8 + h]); else v[h] = fmaf(p1, p2, v[h]);
        }
      }
      lane_scatter<16>(v, lane);
      if ((lane & 1) == 0) red[warp][lane >> 1] = v[0];
      __syncthreads();
      if (tid < 8) {
        const float t0 = warps_sum(red, tid), t1 = warps_sum(red, tid + 8);
        const float r = t1 / __fadd_rn(t0, t1);
        S.of1[mo * 8 + tid] = fmaxf(0.0f, fminf(1.0f, r));
      }
      __syncthreads();
    }
  }
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

int launch_phase_chain(int J, const int32_t* tsel, int nb, const int32_t* nstates, const uint32_t* hvar, int WB,
                       int Kp, const int32_t* npoly, PhaseVars P, PhaseStore S, const ModelConst& mc, cudaStream_t s) {
#define GP_CHAIN(JJ) \
  case JJ: k_phase_chain<JJ><<<2 * nb, CT, 0, s>>>(tsel, nstates, npoly, hvar, WB, Kp, P, S, mc); return GP_OK;
  switch (J) {
    GP_CHAIN(1) GP_CHAIN(2) GP_CHAIN(3) GP_CHAIN(4) GP_CHAIN(5) GP_CHAIN(6) GP_CHAIN(7) GP_CHAIN(8)
    default: return GP_E_ARG;
  }
#undef GP_CHAIN
}

void launch_phase_units(int max_units, const int32_t* tsel, int nb, const int32_t* nstates, const uint32_t* hvar,
                        int WB, int Kp, PhaseVars P, PhaseStore S, uint64_t seed, int iteration,
                        const int32_t* target_ids, cudaStream_t s) {
  if (max_units > 0)
    k_phase_units<<<dim3(max_units < 4096 ? max_units : 4096, nb), 256, 0, s>>>(tsel, nstates, hvar, WB, Kp, P, S, seed,
                                                                               iteration, target_ids);
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

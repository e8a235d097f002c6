// Per-iteration PBWT state selection on the device
// (haplotype_set::matchHapsFromCompressedPBWTSmall, haplotype_set.cpp:317-394,
// with select_common_pd_fg :445-492, select_rare_pd_fg :494-560,
// init_common :562-653, init_rare :655-680, selectK :682-728) followed by the
// state union of conditioning_set::compactSelection (conditioning_set.cpp:96-104).
//
// Given the panel-side prefix/rank arrays (decoded once), every target haplotype's
// sweep over the sites depends only on its own alleles, so a group of lanes runs one
// haplotype. Each selectK push is recorded with the key (site << 1 | phase) so
// that the union can rebuild the per-sample, per-level lists in the reference's
// push order (sites in order, init_common before select_common, haplotypes in
// order, down before up).
#include <algorithm>

#include "select.h"
#include "tc.h"

namespace gp {

namespace {

// Ones before position x: bits and prefix counts in arrays of their own (small
// columns), or as pairs {bits, prefix count} (rank rows).
__device__ __forceinline__ int rank_v(const uint32_t* __restrict__ bits, const uint32_t* __restrict__ pref, int x) {
  return (int)(pref[x >> 5] + __popc(bits[x >> 5] & ((1u << (x & 31)) - 1u)));
}
__device__ __forceinline__ int rank_row(const uint2* row, int x) {
  const uint2 v = row[x >> 5];
  return (int)v.y + __popc(v.x & ~__funnelshift_l(0u, ~0u, x));  // ~0 << (x & 31)
}

// number of entries of the sorted array a[0..n) that are < x (std::lower_bound distance)
__device__ __forceinline__ int lower_count(const int32_t* __restrict__ a, int n, int x) {
  int lo = 0, hi = n;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (a[mid] < x) lo = mid + 1; else hi = mid;
  }
  return lo;
}

// One bulk copy (TMA) of n bytes, a multiple of 16, global to shared memory, both
// 16-byte aligned; completes on the mbarrier.
__device__ __forceinline__ void bulk_load(void* smem, const void* gmem, uint32_t n, uint64_t* bar) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(tc::smem_u32(bar)), "r"(n) : "memory");
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   tc::smem_u32(smem)),
               "l"(gmem), "r"(n), "r"(tc::smem_u32(bar))
               : "memory");
}

// Per-level push lists of one target haplotype, run by the G lanes of its group:
// lane gl owns the levels gl, gl + G, ... The counts live in shared memory while
// the sweep runs and are written back to push_cnt at its end. A lane's pushes to
// its first level wait in registers until the next call, so that the loads of the
// ids are not waited for.
template <int G>
struct Pusher {
  uint32_t* key;
  uint32_t* id;
  int32_t* cnt;  // shared: cnt[level]
  int cap;
  int32_t* overflow;
  int gl;
  uint32_t pend_key;
  uint32_t pend_id0, pend_id1;
  int npend;  // pending pushes of level gl

  __device__ __forceinline__ void push(int level, uint32_t k, uint32_t h) {
    const int c = cnt[level];
    if (c >= cap) {
      *overflow = 1;
      return;
    }
    key[(size_t)level * cap + c] = k;
    id[(size_t)level * cap + c] = h;
    cnt[level] = c + 1;
  }
  __device__ __forceinline__ void flush() {
    if (npend > 0) push(gl, pend_key, pend_id0);
    if (npend > 1) push(gl, pend_key, pend_id1);
    npend = 0;
  }
};

// haplotype_set::selectK (haplotype_set.cpp:682-728); arr == nullptr means the
// identity order. The reference walks down (pbwt_idx, pbwt_idx + 1, ...) and up
// (pbwt_idx - 1, ...) one level at a time and stops a side at its first position
// outside [0, N) or on the other side of ref_rac than allele a; positions on the
// allowed side of ref_rac form an interval, so each side pushes a run whose
// length is known up front, level o from the group's lane o % G (down before up).
template <int G>
__device__ __forceinline__ void select_k(int pbwt_idx, int f, int g, int ref_rac, const uint32_t* __restrict__ arr, int a,
                                      int K, int N, uint32_t key, Pusher<G>& P) {
  int nh_up = 0, nh_down = 0;
  const int d_up = pbwt_idx - f;
  const int d_down = g - pbwt_idx;
  const int k1 = K;
  if (d_up < k1 && d_down < k1) {
    nh_up = d_up;
    nh_down = d_down;
  } else if (d_up >= k1 && d_down >= k1) {
    nh_up = k1;
    nh_down = k1;
  } else if (d_up < k1) {
    nh_down += k1 - d_up;
  } else if (d_down < k1) {
    nh_up += k1 - d_down;
  }
  const bool alt = a != 0;
  int cd = 0, cu = 0;
  if (pbwt_idx >= 0 && pbwt_idx < N && ((pbwt_idx >= ref_rac) == alt)) {
    const int lim = alt ? N : min(ref_rac, N);
    cd = min(nh_down, lim - pbwt_idx);
  }
  const int p = pbwt_idx - 1;
  if (p >= 0 && p < N && ((p >= ref_rac) == alt)) {
    const int lo = alt ? max(ref_rac, 0) : 0;
    cu = min(nh_up, p - lo + 1);
  }
  P.flush();
  int o = P.gl;
  if (o < max(cd, cu)) {
    P.pend_key = key;
    const bool down = o < cd, up = o < cu;
    const int i0 = down ? pbwt_idx + o : p - o;
    P.pend_id0 = arr ? arr[i0] : (uint32_t)i0;
    if (down && up) P.pend_id1 = arr ? arr[p - o] : (uint32_t)(p - o);
    P.npend = (int)down + (int)up;
  }
  for (o += G; o < max(cd, cu); o += G) {
    const uint32_t hd = o < cd ? (arr ? arr[pbwt_idx + o] : (uint32_t)(pbwt_idx + o)) : 0u;
    const uint32_t hu = o < cu ? (arr ? arr[p - o] : (uint32_t)(p - o)) : 0u;
    if (o < cd) P.push(o, key, hd);
    if (o < cu) P.push(o, key, hu);
  }
}

// pbwt_stored groups and random starting positions (haplotype_set.cpp:336-348).
__global__ void k_pbwt_rng(PbwtSelectArgs a) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  const int nw = (a.P.n_com_hq + 32) / 32;
  for (int i = 0; i < nw; ++i) a.stored_bits[i] = 0u;
  StreamCursor g(a.seed, RNG_PBWT, (uint32_t)a.iteration, 0u);
  int loffset = 0;
  for (int i = 0; i < a.nstored; ++i) {
    const uint32_t st = uniform_uint(g, (uint32_t)loffset, (uint32_t)(a.grp[i] - 1));
    a.stored_bits[st >> 5] |= 1u << (st & 31);
    loffset = a.grp[i];
  }
  for (int e = 0; e < a.n_haps; ++e) a.start_idx[e] = (int32_t)uniform_uint(g, 0u, (uint32_t)(a.N - 1));
}

// Per target haplotype, the non-LQ rare sites where it carries the non-major
// allele, as bits: what the init_rare scan of haplotype_set.cpp:655-680 looks
// for, so that the sweep can test a whole run of rare sites at once.
__global__ void k_rare_carriers(PbwtSelectArgs a) {
  const int hp = blockIdx.y;
  const int t = a.hap_target[hp];
  const uint8_t* H = (a.hap_which[hp] ? a.h1 : a.h0) + (size_t)t * a.L;
  for (int wi = blockIdx.x * blockDim.x + threadIdx.x; wi < a.Wc; wi += gridDim.x * blockDim.x) {
    uint32_t bits = 0u;
    const int s0 = wi << 5;
    const int n = min(32, a.L - s0);
    for (int i = 0; i < n; ++i) {
      const int s = s0 + i;
      if (!a.lq[s] && !a.common[s] && H[s] != a.major[s]) bits |= 1u << i;
    }
    a.carry[(size_t)hp * a.Wc + wi] = bits;
  }
}

// Any carrier bit in sites [k0, k1].
__device__ __forceinline__ bool any_carrier(const uint32_t* __restrict__ c, int k0, int k1) {
  const int w0 = k0 >> 5, w1 = k1 >> 5;
  for (int w = w0; w <= w1; ++w) {
    uint32_t v = c[w];
    if (w == w0) v &= ~0u << (k0 & 31);
    if (w == w1) v &= (k1 & 31) == 31 ? ~0u : ((1u << ((k1 & 31) + 1)) - 1u);
    if (v) return true;
  }
  return false;
}

// The per-haplotype bit of every sweep event (PbwtSelectArgs::ebits): the
// allele H[k] at an HQ common site k, or for a run of rare sites [k0, kend] the
// init_rare test (haplotype_set.cpp:655-680), sn > 0 and a carrier bit in the run.
// The sweep reads one word per 32 events, a chunk ahead, instead of a scattered
// byte or carrier load per event on its sequential path. Thread x of a block is
// haplotype blockIdx.x * blockDim.x + x, and blockIdx.y the chunk of 32 events,
// so the event records a warp reads are the same for all its lanes.
__global__ void k_event_bits(PbwtSelectArgs a) {
  const int hp = blockIdx.x * blockDim.x + threadIdx.x;
  if (hp >= a.n_haps) return;
  const int nev = a.P.n_events;
  const int t = a.hap_target[hp];
  const uint8_t* H = (a.hap_which[hp] ? a.h1 : a.h0) + (size_t)t * a.L;
  const uint32_t* carry = a.carry + (size_t)hp * a.Wc;
  for (int c = blockIdx.y; c < a.We; c += gridDim.y) {  // gridDim.y is capped at grid_y_cap <= 65535
    uint32_t bits = 0u;
    const int n = min(32, nev - (c << 5));
    for (int i = 0; i < n; ++i) {
      const int e = (c << 5) + i;
      const int4 r0 = a.P.events[2 * e];
      const int4 r1 = a.P.events[2 * e + 1];
      bool b;
      if (!(r0.x & (1 << 30))) b = H[r0.x] != 0;
      else b = r1.x > 0 && any_carrier(carry, r0.x & ~(1 << 30), r0.z);
      if (b) bits |= 1u << i;
    }
    a.ebits[(size_t)hp * a.We + c] = bits;
  }
}

// The sweep: one warp per HPW target haplotypes (1, 2, 4 or 8, chosen by the
// autotuner), G = 32 / HPW lanes per haplotype. A haplotype's chain over the events
// (non-LQ common sites and runs of rare sites, in site order) is bound by the
// latency of its dependent integer instructions: each event's interval depends on
// the previous one's. All lanes of a group run the chain (the three rank lookups
// of an event are independent of one another); the levels of a selectK are spread
// over the group's lanes, and their loads are not waited for.
//
// The haplotypes of a warp walk the event list in step; what only some of them do
// (an empty interval, a stored site, a carried rare run) branches per group.
// Shared memory per warp holds
//   ring    kRankStages stages of rows_per consecutive rank rows, one bulk copy
//           each, kRankStages - 1 stages ahead (row l: pairs {bits, prefix count} of
//           the V ranks of select_common_pd_fg, then of the small-PBWT position
//           ranks of init_common), and an mbarrier per stage;
//   evbuf   two chunks of 32 event records (the next chunk is loaded one chunk ahead);
//   scnt    the per-level push counts of each haplotype.
// Without RING the rows are read from global memory (panels whose rows do not fit
// in shared memory). Waits are bounded; a time-out sets the overflow flag to 2.
// Measured per sweep: 20,000 events, 1,000 haplotypes, one target 11.0 -> 4.1 ms;
// 54,000 events, 10,000 haplotypes, 256 targets 25.8 -> 10.6 ms (2 per warp; 18.3, 11.2
// and 12.2 ms for 1, 4 and 8, as every warp reads all rank rows once). Before, the rows
// came by one 16-byte copy per lane and 512 bytes, addresses and shapes were run-time
// values, and a selectK waited for its ids.
constexpr int kRankStages = 3;

// Group q of rank rows goes to stage q % kRankStages and completes the phase of this
// parity there. While group g is waited for, the groups g .. g + kRankStages - 1 are
// requested and not waited for (as far as there are any).
__host__ __device__ constexpr uint32_t rank_parity(int q) { return (uint32_t)(q / kRankStages) & 1u; }

// The sweep's own stage and parity, and its requests, over n groups.
constexpr bool ring_agrees(int n) {
  int stage = kRankStages - 1, requested[kRankStages] = {};
  uint32_t parity = 1u;
  for (int st = 0; st < kRankStages && st < n; ++st) requested[st] = 1;
  for (int g = 0; g < n; ++g) {
    if (g > 0 && g + kRankStages - 1 < n) ++requested[stage];
    if (++stage == kRankStages) {
      stage = 0;
      parity ^= 1u;
    }
    if (stage != g % kRankStages || parity != rank_parity(g)) return false;
    for (int q = g; q < g + kRankStages && q < n; ++q)  // what a time-out has to wait for: every stage's last request
      if (rank_parity(q) != ((uint32_t)(requested[q % kRankStages] - 1) & 1u)) return false;
  }
  return true;
}
static_assert(ring_agrees(1) && ring_agrees(2) && ring_agrees(3) && ring_agrees(4) && ring_agrees(17), "rank row stages");

template <int HPW, bool RING>
__global__ void __launch_bounds__(32, 1) k_pbwt_sweep(PbwtSelectArgs a, int rows_per) {
  constexpr int G = 32 / HPW;
  extern __shared__ __align__(16) uint32_t smem[];
  __shared__ uint64_t bars[kRankStages];
  const int lane = threadIdx.x & 31;
  const int grp = lane / G, gl = lane % G;
  const bool act = blockIdx.x * HPW + grp < a.n_haps;  // idle groups repeat the last haplotype and record nothing
  const int hp = min((int)(blockIdx.x * HPW + grp), a.n_haps - 1);
  const DevPbwt& P = a.P;
  const int R = P.R, ncom = P.n_com_hq, nev = P.n_events;
  const int N = a.N, K = a.depth;
  const int stage_words = RING ? rows_per * R : 0;
  uint32_t* ring = smem;
  int4* evbuf = reinterpret_cast<int4*>(smem + kRankStages * stage_words);  // [2][32][2]
  int32_t* scnt = reinterpret_cast<int32_t*>(evbuf + 2 * 32 * 2) + grp * K;  // [HPW][K]

  // stage st takes the rows [rows_per * g, rows_per * (g + 1)) of group g = st modulo kRankStages
  auto load_rows = [&](int first, int st) {
    if (first < ncom)
      bulk_load(ring + st * stage_words, P.vrow + (size_t)first * R, (uint32_t)(min(rows_per, ncom - first) * R * 4),
                &bars[st]);
  };
  if (RING && lane == 0) {
    for (int st = 0; st < kRankStages; ++st) tc::mbar_init(&bars[st], 1);
    tc::fence_mbar_init();
    for (int st = 0; st < kRankStages; ++st) load_rows(st * rows_per, st);
  }
  // Event chunk c (32 records) goes to evbuf[c & 1]; chunk c + 1 is loaded when chunk c starts.
  auto load_chunk = [&](int c) {
    const int en = (c << 5) + lane;
    if (en < nev) {
      evbuf[((c & 1) * 32 + lane) * 2] = P.events[2 * en];
      evbuf[((c & 1) * 32 + lane) * 2 + 1] = P.events[2 * en + 1];
    }
  };
  load_chunk(0);
  load_chunk(1);

  const int t = a.hap_target[hp];
  const uint8_t* H = (a.hap_which[hp] ? a.h1 : a.h0) + (size_t)t * a.L;
  // event bits of the current chunk and of the next one
  const uint32_t* eb = a.ebits + (size_t)hp * a.We;
  uint32_t ebw = a.We > 0 ? eb[0] : 0u;
  uint32_t ebn = a.We > 1 ? eb[1] : 0u;
  // stored sites l & ~31 .. and the next 32
  uint32_t sbw = 0u, sbn = a.stored_bits[0];
  Pusher<G> pu;
  pu.key = a.push_key + (size_t)hp * K * a.cap;
  pu.id = a.push_id + (size_t)hp * K * a.cap;
  pu.cnt = scnt;
  pu.cap = a.cap;
  pu.overflow = a.overflow;
  pu.gl = gl;
  pu.pend_key = pu.pend_id0 = pu.pend_id1 = 0u;
  pu.npend = 0;
  for (int o = gl; o < K; o += G) scnt[o] = 0;
  int idx = a.start_idx[hp], f = 0, g = N;
  int sidx = 0, fs = 0, gs = 0;  // the same in the run's small PBWT
  int last_reset = 0, last_rare = 0;
  int tar = a.tar_hap[hp];
  bool in_rare = false;
  int prev_ref_com = 0;
  const float half_mod = a.modulo / 2.0f;
  const float fifth_mod = a.modulo / 5.0f;
  const int half = R >> 1;
  const uint32_t* row = RING ? smem : P.vrow;  // rank row of the next HQ common site
  int in_stage = rows_per - 1;                // its place in its stage
  int stage = kRankStages - 1;                // its stage, and the parity to wait for
  uint32_t parity = 1u;
  int next_rows = (kRankStages - 1) * rows_per;  // first row of the stage to request next
  bool failed = false;
  __syncwarp();
  int4 r0 = evbuf[0], r1 = evbuf[1];

#pragma unroll 2
  for (int e = 0; e < nev; ++e) {
    if ((e & 31) == 0 && e > 0) {
      const int c = e >> 5;
      load_chunk(c + 1);  // chunk c - 1 is no longer read: its last record was read before the last __syncwarp
      ebw = ebn;
      ebn = c + 1 < a.We ? eb[c + 1] : 0u;
    }
    const bool ebit = (ebw >> (e & 31)) & 1u;
    const int4 q0 = r0, q1 = r1;
    __syncwarp();
    {
      const int4* nx = evbuf + (((e + 1) & 63) * 2);  // the record after the last one is read and not used
      r0 = nx[0];
      r1 = nx[1];
    }
    if (!(q0.x & (1 << 30))) {
      // ---------------- HQ common site ----------------
      const int k = q0.x, l = q0.y, ref = q0.z;
      if (RING && ++in_stage == rows_per) {
        // The stage before is free: every lane is past its last row (the __syncwarp above).
        if (lane == 0 && l > 0) load_rows(next_rows, stage);
        next_rows += rows_per;
        in_stage = 0;
        if (++stage == kRankStages) {
          stage = 0;
          parity ^= 1u;
        }
        if (!tc::mbar_wait(&bars[stage], parity)) {
          failed = true;
          break;
        }
        row = smem + stage * stage_words;
      }
      if (q1.z) {  // init_common
        const int sn = q1.x;
        const uint2* srow = reinterpret_cast<const uint2*>(row + half);
        int nidx, nf, ng;
        if (in_rare) {
          nidx = N - sn + sidx;
          nf = last_reset >= last_rare ? 0 : N - sn + fs;
          ng = N - sn + gs;
        } else {
          // numbers of small-PBWT positions below f, g and idx: ranks in the row's second part
          nidx = idx - rank_row(srow, idx);
          nf = f - rank_row(srow, f);
          ng = g - rank_row(srow, g);
        }
        if (ng <= nf) {
          const uint32_t* a_pre = l > 0 ? P.a_after + (size_t)(l - 1) * N : nullptr;
          const int prev_site = q1.w;  // common2tot indexed by the HQ count, as the reference does
          if (act && (in_rare || __fsub_rn(P.cm_pos[prev_site], P.cm_pos[last_reset]) > fifth_mod))
            select_k<G>(idx, f, g, prev_ref_com, a_pre, tar, K, N, (uint32_t)(k << 1), pu);
          nf = 0;
          ng = in_rare ? N : N - sn;
          last_reset = in_rare ? k - 1 : prev_site;
        }
        idx = nidx;
        f = nf;
        g = ng;
      }
      // select_common_pd_fg at HQ common site l
      const uint2* vrow = reinterpret_cast<const uint2*>(row);
      row += R;
      const int vi = rank_row(vrow, idx), vf = rank_row(vrow, f), vg = rank_row(vrow, g);
      const int al = ebit ? 1 : 0;  // H[k]
      if ((l & 31) == 0) {
        sbw = sbn;
        if (l + 32 < ncom) sbn = a.stored_bits[(l >> 5) + 1];
      }
      const bool stored = (sbw >> (l & 31)) & 1u;
      const int nidx = al ? ref + vi : idx - vi;
      int nf = al ? ref + vf : f - vf;
      int ng = al ? ref + vg : g - vg;
      if (ng <= nf || stored) {
        if (ng <= nf) {
          const int km1 = k > 0 ? k - 1 : 0;
          if (act && (stored || __fsub_rn(P.cm_pos[km1], P.cm_pos[last_reset]) > half_mod)) {
            const int bid = q1.y;
            const uint32_t* a_pre = l > 0 ? P.a_after + (size_t)(l - 1) * N : nullptr;
            const uint32_t* b_arr = bid >= 0 ? P.merged + (size_t)bid * N : (bid == -1 ? a_pre : nullptr);
            select_k<G>(idx, f, g, prev_ref_com, b_arr, tar, K, N, (uint32_t)((k << 1) | 1), pu);
          }
        } else if (act) {
          select_k<G>(nidx, nf, ng, ref, P.a_after + (size_t)l * N, al, K, N, (uint32_t)((k << 1) | 1), pu);
        }
        nf = al * ref;
        ng = al * N + (1 - al) * ref;
        last_reset = k;
      }
      idx = nidx;
      f = nf;
      g = ng;
      tar = al;
      prev_ref_com = ref;
    } else {
      // ---------------- run of rare sites [k0, kend] ----------------
      // init_rare: is this haplotype in rareTarHaps for the run?
      in_rare = ebit;  // sn > 0 and a carrier bit in [k0, kend]
      // Nothing happens at the run's sites for a haplotype outside rareTarHaps.
      if (in_rare) {
        const int k0 = q0.x & ~(1 << 30), kend = q0.z, so = q0.w, sn = q1.x;
        const int32_t* sm = P.asidx + so;
        int fsn = lower_count(sm, sn, f);
        int gsn = lower_count(sm, sn, g);
        if (gsn <= fsn) {
          fsn = 0;
          gsn = sn;
          last_reset = k0;
        }
        sidx = lower_count(sm, sn, idx);
        fs = fsn;
        gs = gsn;
        for (int k = k0; k <= kend; ++k) {
          const int info = P.site_info[k];
          if ((info & 3) == SK_LQ) continue;
          const int r = info >> 2;
          const int ref = a.major[k] ? (int)P.cref[k] : sn - (int)a.calt[k];
          const uint32_t* vb = P.svbits + P.svoff[r];
          const uint32_t* vp = P.svpref + (P.svoff[r] + r);
          const int vi = rank_v(vb, vp, sidx), vf = rank_v(vb, vp, fs), vg = rank_v(vb, vp, gs);
          const bool car = H[k] != a.major[k];
          if (car) last_rare = k;
          sidx = car ? ref + vi : sidx - vi;
          fs = car ? ref + vf : fs - vf;
          gs = car ? ref + vg : gs - vg;
          if (gs <= fs) {
            fs = car ? ref : 0;
            gs = car ? sn : ref;
            last_reset = k;
          }
        }
      }
    }
  }
  if (RING && failed) {
    // The copies requested and not waited for may still be under way: wait for each, bounded
    // as well, before the memory is given up. The lists so far are in order for the union.
    *a.overflow = 2;
    for (int q = next_rows / rows_per - kRankStages; q * rows_per < min(next_rows, ncom); ++q)
      tc::mbar_wait(&bars[q % kRankStages], rank_parity(q));
  }
  if (!act) return;
  pu.flush();
  for (int o = gl; o < K; o += G) a.push_cnt[(size_t)hp * K + o] = scnt[o];
  if (gl == 0) a.tar_hap[hp] = (uint8_t)tar;
}

// conditioning_set::compactSelection union (conditioning_set.cpp:96-104): levels
// in order, each level from its last push backwards, until Kpbwt states. A warp per
// target. A haplotype's keys do not decrease along a level, so the two haplotypes'
// lists are merged 32 pushes at a time: a push's place is its own index plus the pushes
// of the other list that go before it. Bound by the latency of the loads, two in a row
// per 32 pushes (a thread per target, two in a row per push: 256 targets
// 1.2 ms, 0.1 now).
__global__ void __launch_bounds__(32) k_pbwt_union(PbwtSelectArgs a) {
  constexpr uint32_t kAll = 0xffffffffu;
  __shared__ uint32_t merged[32];
  const int t = blockIdx.x, lane = threadIdx.x;
  const int N = a.N, K = a.depth, cap = a.cap;
  const int W = (N + 31) / 32;
  uint32_t* bm = a.bitmap + (size_t)t * W;
  for (int i = lane; i < W; i += 32) __stcg(&bm[i], 0u);
  __threadfence();
  __syncwarp();
  const int kmax = a.kpbwt[t];
  const int h0 = a.target_hap0[t], nh = a.target_nhap[t];
  int count = 0;
  for (int lv = 0; lv < K && count < kmax; ++lv) {
    int p[2] = {-1, -1};
    const uint32_t* keys[2] = {nullptr, nullptr};
    const uint32_t* ids[2] = {nullptr, nullptr};
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int hp = h0 + j;
      if (j < nh) p[j] = a.push_cnt[(size_t)hp * K + lv] - 1;
      keys[j] = a.push_key + ((size_t)hp * K + lv) * cap;
      ids[j] = a.push_id + ((size_t)hp * K + lv) * cap;
    }
    while (count < kmax && (p[0] >= 0 || p[1] >= 0)) {
      uint32_t key[2] = {0u, 0u}, id[2] = {0u, 0u};
      int n[2], before[2] = {0, 0};  // loaded pushes of each list; of the other list, those before this lane's
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        n[j] = min(32, p[j] + 1);
        if (lane < n[j]) {
          key[j] = keys[j][p[j] - lane];
          id[j] = ids[j][p[j] - lane];
        }
      }
#pragma unroll
      for (int i = 0; i < 6; ++i) {
        const int step = i < 5 ? 16 >> i : 1;
        const uint32_t k1 = __shfl_sync(kAll, key[1], before[0] + step - 1);
        const uint32_t k0 = __shfl_sync(kAll, key[0], before[1] + step - 1);
        if (before[0] + step <= n[1] && k1 >= key[0]) before[0] += step;  // of equal keys the second haplotype's first
        if (before[1] + step <= n[0] && k0 > key[1]) before[1] += step;
      }
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const int at = lane + before[j];
        const bool take = lane < n[j] && at < 32;
        if (take) merged[at] = id[j];
        p[j] -= __popc(__ballot_sync(kAll, take));
      }
      __syncwarp();
      const bool in = lane < min(32, n[0] + n[1]);
      const uint32_t h = in ? merged[lane] : 0x80000000u | lane;
      const uint32_t m = 1u << (h & 31);
      const bool first = __ffs(__match_any_sync(kAll, h)) - 1 == lane;
      const bool fresh = in && first && !(__ldcg(&bm[in ? h >> 5 : 0]) & m);
      const uint32_t all = __ballot_sync(kAll, fresh);
      const int at = count + __popc(all & ((1u << lane) - 1u));
      if (fresh && at < kmax) {
        atomicOr(&bm[h >> 5], m);
        if (a.union_rank) a.union_rank[(size_t)t * N + h] = (lv << 16) | min(at, 0xFFFF);
      }
      count = min(kmax, count + __popc(all));
      __threadfence();
      __syncwarp();
    }
  }
  int k = 0;
  for (int i0 = 0; i0 < W; i0 += 32) {
    const int i = i0 + lane;
    uint32_t w = i < W ? __ldcg(&bm[i]) : 0u;
    int end = __popc(w);
    const int own = end;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(kAll, end, o);
      if (lane >= o) end += v;
    }
    for (int q = k + end - own; w; ++q, w &= w - 1)
      if (q < a.Kp) a.states[(size_t)t * a.Kp + q] = (uint32_t)(i * 32 + __ffs(w) - 1);
    k += __shfl_sync(kAll, end, 31);
  }
  if (lane == 0) a.nstates[t] = k;
}

}  // namespace

template <int HPW>
static void launch_sweep(const PbwtSelectArgs& a, cudaStream_t s) {
  // Stages of 4, 2 or 1 rank rows, within 96 KB. Larger panels (above some 65,000 haplotypes)
  // read from memory: there three longer rows a stage leave one warp per SM, and 256 targets of
  // 80,000 haplotypes took 3.3, 2.0 or 1.27 ms (1, 2, 4 per warp) against 0.94, 1.08 or 1.22.
  constexpr int kLimit = 200 << 10;
  const size_t row_bytes = (size_t)a.P.R * 4, fixed = 2 * 32 * 2 * 16 + (size_t)a.depth * HPW * 4;
  int rows = 4;
  while (rows > 0 && kRankStages * rows * row_bytes > (96u << 10)) rows >>= 1;
  const int grid = (a.n_haps + HPW - 1) / HPW;
  if (rows > 0) {
    const size_t smem = kRankStages * rows * row_bytes + fixed;
    if (smem > (48u << 10)) set_smem_limit_once<k_pbwt_sweep<HPW, true>>(kLimit);
    k_pbwt_sweep<HPW, true><<<grid, 32, smem, s>>>(a, rows);
  } else {
    if (fixed > (48u << 10)) set_smem_limit_once<k_pbwt_sweep<HPW, false>>(kLimit);  // very deep lists
    k_pbwt_sweep<HPW, false><<<grid, 32, fixed, s>>>(a, 1);
  }
}

cudaError_t launch_pbwt_sweep(const PbwtSelectArgs& a, int hpw, cudaStream_t s) {
  if (hpw == 1) launch_sweep<1>(a, s);
  else if (hpw == 2) launch_sweep<2>(a, s);
  else if (hpw == 4) launch_sweep<4>(a, s);
  else launch_sweep<8>(a, s);
  return cudaGetLastError();
}

cudaError_t launch_pbwt_select(const PbwtSelectArgs& a, int hpw, cudaStream_t s) {
  launch_pbwt_prepare(a, s);
  const cudaError_t e = launch_pbwt_sweep(a, hpw, s);
  if (e != cudaSuccess) return e;  // without the sweep there are no lists to unite
  k_pbwt_union<<<a.n_targets, 32, 0, s>>>(a);
  return cudaGetLastError();
}

void launch_pbwt_prepare(const PbwtSelectArgs& a, cudaStream_t s) {
  k_pbwt_rng<<<1, 32, 0, s>>>(a);
  k_rare_carriers<<<dim3((a.Wc + 127) / 128, a.n_haps), 128, 0, s>>>(a);
  const int ycap = std::max(1, std::min(a.grid_y_cap, 65535));
  if (a.We > 0) k_event_bits<<<dim3((a.n_haps + 127) / 128, std::min(a.We, ycap)), 128, 0, s>>>(a);
}

}  // namespace gp

// Device data of the phasing HMM (kernels_phase.cu).
#pragma once
#include "internal.h"

namespace gp {

constexpr int kPhaseThreads = 256;  // states per j of a chain, over 8 virtual warps
// VAR codes: 0..2 peak het of type n_het % 3, VT_HOM peak hom, VT_FLAT flat het
// (VAR_PEAK_HET / VAR_PEAK_HOM / VAR_FLAT_HET, phasing_hmm.h:40-42); bit 3 = VAR_ALT.
constexpr int VT_HOM = 3;
constexpr int VT_FLAT = 4;

// Per batch entry b: arrays of stride L (VAR entries), L+2 (segments).
struct PhaseVars {
  int32_t* rel;        // VAR_REL: poly index
  uint8_t* code;       // type | alt << 3
  int32_t* seg;        // segment of the entry
  int32_t* miss;       // flat-het index or -1
  int32_t* miss_rel;   // VAR_REL of each flat het
  int32_t* seg_start;  // first entry of each segment, [nseg] = nvar
  float* yt_prev;      // transition from the previous VAR site (0 for the first)
  float* yt_next;      // transition to the next VAR site (0 for the last)
  uint8_t* flags;      // bit0: first entry of its segment, bit1: last entry of its segment
  // The fields the sweeps read per entry, packed into 16 bytes per direction:
  // x = rel | code << 24 | flags << 28, y = seg, z = miss, w = bits of the
  // transition to the next entry (recb, backward) or from the previous one (recf).
  int4* recb;
  int4* recf;
  int32_t* nvar;
  int32_t* nseg;
  int32_t* nmiss;
  // Per-entry stride of the arrays above: the batch's largest polymorphic-site count (VAR sites are a subset).
  int lv;
};

// Per entry b: rows of 8 floats per state in the pool at pool_off[b], [nseg][K][8] backward messages at segment
// starts, [nmiss][K][8] backward messages at flat hets, then the forward messages at segment ends and at flat
// hets. Segment and flat-het arrays of all entries are packed: entry b's segments start at seg_off[b] (seg_total
// in all), its flat hets at miss_off[b]; sums have a backward half and, seg_total or miss_total further on, a
// forward half.
struct PhaseStore {
  float* pool;
  const int64_t* pool_off;
  const int64_t* seg_off;
  const int64_t* miss_off;
  int64_t seg_total, miss_total;
  float* seg_sum;        // [2][seg_total][8] sums of the stored messages per hypothesis
  float* seg_tot;        // [2][seg_total] their totals
  float* miss_sum;       // [2][miss_total][8]
  float* of1;            // imputeProbOf1s [miss_total][8]
  uint32_t* next;        // [seg_total] drawn successor of each diplotype (3 bits each) and error bits from bit 24
  int32_t* dip;          // [seg_total] dip_sampled
  int32_t* err;          // [b] nonzero when a diplotype draw saw an invalid sum
  const int32_t* order;  // [nb] batch entries in launch order (heaviest first)
};

void launch_build_vars(const int32_t* tsel, int nb, const int32_t* poly, const int32_t* npoly, const uint8_t* h0,
                       const uint8_t* h1, const uint8_t* flat, const uint8_t* lq, int L, PhaseVars V,
                       cudaStream_t s);
// Per-VAR transition records of all nb entries (before the phasing launches).
void launch_var_records(const int32_t* tsel, int nb, const int32_t* poly, int L, const double* cm,
                        const ModelConst& mc, PhaseVars V, cudaStream_t s);
// The backward and forward chains of the nb entries S.order[0 .. nb), all with
// 256 (J - 1) < K <= 256 J states (S.order may point into a longer order). narrow:
// two warps a chain instead of four, for J <= kPhaseNarrowJ.
constexpr int kPhaseNarrowJ = 5;
// Chains of class J that are resident on an SM together (their registers are bounded to that).
constexpr int phase_chains_per_sm(int J, bool narrow) {
  return narrow ? (J <= 3 ? 6 : 4) : J <= 2 ? 5 : J <= 4 ? 4 : J <= 5 ? 3 : 2;
}
int launch_phase_chain(int J, bool narrow, const int32_t* tsel, int nb, const int32_t* nstates, const uint32_t* hvar,
                       int WB, int Kp, const int32_t* npoly, PhaseVars P, PhaseStore S, const ModelConst& mc,
                       cudaStream_t s);
// After the chains, for entries of any K: the units. max_units: the largest count of
// segment boundaries and flat hets of an entry; bit J of narrow: the chains of class J
// ran narrow.
int launch_phase_units(int max_units, uint32_t narrow, const int32_t* tsel, int nb, const int32_t* nstates,
                       const uint32_t* hvar, int WB, int Kp, PhaseVars P, PhaseStore S, uint64_t seed, int iteration,
                       const int32_t* target_ids, cudaStream_t s);
// After the units: the diplotype chains.
void launch_phase_draw(const int32_t* tsel, int nb, PhaseVars P, PhaseStore S, uint64_t seed, int iteration,
                       const int32_t* target_ids, cudaStream_t s);
void launch_phase_writeback(const int32_t* tsel, int nb, const int32_t* poly, const int32_t* polyidx, int L,
                            PhaseVars V, PhaseStore S, const ModelConst& mc, uint64_t seed, int iteration,
                            const int32_t* target_ids, uint8_t* h0, uint8_t* h1, cudaStream_t s);

}  // namespace gp

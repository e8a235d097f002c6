// Internal declarations shared by the CUDA translation units of libglimpse_b200.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>
#include <string>
#include <vector>

#include "../../include/glimpse_b200.h"
#include "replay_rng.h"

namespace gp {

constexpr int kWarp = 32;

#ifdef __CUDACC__
// Two floats in one 64-bit register pair (lo = first); the packed mul / add /
// fma (sm_100a) round each element exactly as the scalar instructions do.
typedef unsigned long long f2;
__device__ __forceinline__ f2 f2_pack(float lo, float hi) {
  f2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void f2_unpack(f2 v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ f2 f2_fma(f2 a, f2 b, f2 c) {
  f2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ f2 f2_mul(f2 a, f2 b) {
  f2 d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ f2 f2_add(f2 a, f2 b) {
  f2 d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
#endif
constexpr int kImputeThreads = 256;           // threads per haplotype in the imputation HMM
constexpr int kImputeStatesPerThread = 8;     // registers per thread for owned states
constexpr int kMaxStates = kImputeThreads * kImputeStatesPerThread;  // 2048
constexpr int kHaps = 8;                      // HAP_NUMBER (phasing_hmm.h:38)

// Status carried out of host helpers.
struct Status {
  int code = GP_OK;
  std::string msg;
};

// A kernel's dynamic shared-memory limit, set once per device (the attribute is
// per device; contexts may sit on different devices). F is the kernel.
template <auto F>
cudaError_t set_smem_limit_once(int bytes) {
  static std::atomic<uint64_t> done{0};  // bit d: set on device d
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const uint64_t bit = 1ull << (dev & 63);
  if (dev < 64 && (done.load(std::memory_order_acquire) & bit)) return cudaSuccess;
  e = cudaFuncSetAttribute(F, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e == cudaSuccess && dev < 64) done.fetch_or(bit, std::memory_order_acq_rel);
  return e;
}

// Host-side fault injection for tests: true when GLIMPSE_B200_FAIL_ALLOC=n is
// set and this is the n-th buffer growth since it was read (the variable is
// re-read whenever its value changes). The growth then reports
// cudaErrorMemoryAllocation without calling cudaMalloc.
bool inject_alloc_failure();

// Growable device buffer (bytes); contents are not preserved on growth.
struct DevBuf {
  void* ptr = nullptr;
  size_t cap = 0;
  cudaError_t ensure(size_t bytes) {
    if (bytes <= cap) return cudaSuccess;
    if (ptr) cudaFree(ptr);
    ptr = nullptr;
    cap = 0;
    if (inject_alloc_failure()) return cudaErrorMemoryAllocation;
    size_t want = bytes + bytes / 8 + 256;
    cudaError_t e = cudaMalloc(&ptr, want);
    if (e == cudaSuccess) cap = want;
    return e;
  }
  void release() {
    if (ptr) cudaFree(ptr);
    ptr = nullptr;
    cap = 0;
  }
  template <class T> T* as() const { return static_cast<T*>(ptr); }
};

// Panel resident in device memory.
struct DevPanel {
  int N = 0, L = 0, n_com = 0, n_com_hq = 0, W = 0;  // W: 32-bit words per haplotype over common rows
  double* cm = nullptr;
  uint8_t* lq = nullptr;
  uint8_t* common = nullptr;
  uint8_t* major = nullptr;
  uint32_t* cref = nullptr;
  uint32_t* calt = nullptr;
  int32_t* comrow = nullptr;       // site -> common row, -1 for rare
  uint32_t* refT = nullptr;        // [N][W] haplotype-major bits over common rows (bit r%32 of word r/32)
  int64_t* shap_off = nullptr;     // [N+1]
  int32_t* shap_sites = nullptr;   // rare sites carrying the non-major allele, per haplotype
  int64_t shap_nnz = 0;
  int64_t* svar_off = nullptr;     // [L+1] SvarRef CSR
  int32_t* svar_haps = nullptr;
};

// Per-batch scratch for the imputation path (sized for n haplotypes).
struct ImputeWork {
  int n = 0, L = 0, Kp = 0, WB = 0;  // WB: 32-site blocks per haplotype (upper bound)
  DevBuf states, nstates, states_off;
  DevBuf mark, polyidx, poly, npoly;
  DevBuf hvar, em, tr, fl;
  DevBuf rows, row_off, fac;  // kept rows of the chains and their offsets, the factors of every site
  DevBuf order;  // [n] haplotypes in decreasing order of poly sites (chain launch order); ptr null: identity
  DevBuf hl, hp, flat;
};

// Scratch of the phasing HMM.
struct PhaseWork {
  DevBuf rel, code, seg, miss, miss_rel, seg_start, counts, ytp, ytn, vflags, recb, recf;
  DevBuf pool;  // the stored messages of one chunk of entries
  DevBuf offs, seg_sum, seg_tot, miss_sum, of1, next, dip, err, order;
  std::vector<DevBuf*> all() {
    return {&rel, &code, &seg, &miss, &miss_rel, &seg_start, &counts, &ytp, &ytn, &vflags, &recb, &recf, &pool,
            &offs, &seg_sum, &seg_tot, &miss_sum, &of1, &next, &dip, &err, &order};
  }
};

// Model constants derived from gp_config the way the reference derives them
// (conditioning_set.cpp:27-37, caller_initialise.cpp:150-153).
struct ModelConst {
  float ed_imp, ee_imp, ed_phs, ee_phs, min_gl;
  double nrho, one_l;
};

// Kernel launchers (kernels_impute.cu).
void launch_mark_poly(const DevPanel& P, ImputeWork& w, cudaStream_t s);
void launch_compact_poly(const DevPanel& P, ImputeWork& w, cudaStream_t s);
void launch_build_hvar(const DevPanel& P, ImputeWork& w, cudaStream_t s);
void launch_site_records(const DevPanel& P, const ModelConst& mc, ImputeWork& w, const float* hl,
                         const uint8_t* flat, cudaStream_t s);
// Sites between kept rows of a chain (a divisor of 32): two rows, one per direction.
constexpr int kRowSites = 16;
// Forward and backward chains of the haplotypes order[first .. first + count)
// (count < 0: all n), all with impute_groups(K) = J, cpc chains per CTA (1, 2 or 4).
int launch_impute_chain(int J, ImputeWork& w, cudaStream_t s, int first = 0, int count = -1, int cpc = 1);
// After the chains, for haplotypes of any K with at most max_poly polymorphic
// sites: prob_hid of every site into hp.
int launch_impute_block(int max_poly, ImputeWork& w, float* hp, cudaStream_t s, int first = 0, int count = -1);
// Rows of 128 states that a chain of K states runs (the J of launch_impute_chain).
int impute_groups(int K);

// The checkpointed modes (kernels_impute_ckpt.cu). A haplotype is split at site M = 32 mblk,
// about np / 2. Both chains first run their own half ([0, M) forward, [M, np) backward) and
// keep checkpoints of it: a row per 16 sites (FP32), or one per 32 rounded to BF16. Then they
// run the other's half in windows, whose posteriors are formed window by window, beside the
// chains of the next one: only two windows' rows exist at a time. All of a haplotype's rows
// lie together, of Ks states each.
struct CkptLayout {
  int nrow, nblk, mblk;  // blocks of 16 and of 32 sites, blocks of 32 before M
  int Ks;                // row stride: states rounded up to 128
  // blocks of 32 of a window, and its rows' place (floats) for even windows; odd ones lie behind: in
  // [M, np), run forward, and in [0, M), run backward
  int wlen0, wlen1, wrows0, wrows1;
  int64_t win0, win1;
  int64_t state, total;  // floats: the chains' states between launches (row and sum, two rows each), all
};
#ifdef __CUDACC__
__host__ __device__
#endif
inline CkptLayout ckpt_layout(int np, int K, bool bf16, int windows) {
  CkptLayout a;
  a.nrow = (np + 15) / 16;
  a.nblk = (np + 31) / 32;
  a.mblk = np / 64;
  a.Ks = (K + 127) / 128 * 128;
  a.wlen0 = (a.nblk - a.mblk + windows - 1) / windows;
  a.wlen1 = (a.mblk + windows - 1) / windows;
  a.state = (int64_t)(bf16 ? (a.nblk + 1) / 2 : a.nrow) * a.Ks;
  // a window's rows: those of the chain, and in BF16 mode the recomputed ones of the other direction
  a.wrows0 = (bf16 ? 4 : 2) * a.wlen0;
  a.wrows1 = (bf16 ? 4 : 2) * a.wlen1;
  a.win0 = a.state + 4 * a.Ks;
  const int kept = windows > 1 ? 2 : 1;
  a.win1 = a.win0 + (int64_t)kept * a.wrows0 * a.Ks;
  a.total = a.win1 + (int64_t)kept * a.wrows1 * a.Ks;
  return a;
}
// The rows (floats) of window w in half 0 or 1.
#ifdef __CUDACC__
__host__ __device__
#endif
inline int64_t ckpt_window_rows(const CkptLayout& a, int half, int w) {
  return half == 0 ? a.win0 + (w & 1 ? (int64_t)a.wrows0 * a.Ks : 0) : a.win1 + (w & 1 ? (int64_t)a.wrows1 * a.Ks : 0);
}
// The blocks [lo, hi) of 32 sites of window w in [M, np) (half 0) or [0, M) (half 1).
#ifdef __CUDACC__
__host__ __device__
#endif
inline void ckpt_window(const CkptLayout& a, int half, int w, int& lo, int& hi) {
  if (half == 0) {
    lo = a.mblk + w * a.wlen0;
    hi = lo + a.wlen0 < a.nblk ? lo + a.wlen0 : a.nblk;
  } else {
    hi = a.mblk - w * a.wlen1;
    lo = hi - a.wlen1 > 0 ? hi - a.wlen1 : 0;
  }
}
// For the haplotypes order[first .. first + count), all with 256 (J - 1) < K <= 256 J: the
// chains over their own halves (win < 0) or window win; asum: [n][32 WB]. Then the
// posteriors of a window of at most wlen blocks of 32 in either half (launch_ckpt_posteriors
// after the rows that BF16 mode recomputes).
int launch_ckpt_chain(int J, bool bf16, bool few, int windows, int win, ImputeWork& w, float* asum, cudaStream_t s,
                      int first, int count);
int launch_ckpt_window(int J, bool bf16, int windows, int win, int wlen, ImputeWork& w, float* hp, cudaStream_t s,
                       int first, int count);
int launch_ckpt_posteriors(bool bf16, int windows, int win, int wlen, ImputeWork& w, float* hp, cudaStream_t s,
                           int first, int count);
// The FP64 log-likelihood of every haplotype from its AlphaSums.
void launch_ckpt_loglik(ImputeWork& w, const float* asum, double* loglik, cudaStream_t s);
void launch_impute_finish(const DevPanel& P, const ModelConst& mc, ImputeWork& w, const float* hl,
                        const uint8_t* flat, float* hp, cudaStream_t s);

}  // namespace gp

/*
 * ORACLE — test infrastructure only. Never linked into the product library.
 *
 * Plain-C restatement of the haploid Li-Stephens imputation HMM of
 * GLIMPSE2_phase, in double precision (the FP64 reference for precision
 * reporting) and in single precision with sequential sums (checked against the
 * reference's own compiled code within 1e-5):
 *   - conditioning set: polymorphic sites and Hvar bits
 *     (phase/src/containers/conditioning_set.cpp:123-182),
 *   - transitions (conditioning_set.cpp:184-196),
 *   - emissions (phase/src/models/imputation_hmm.cpp:124-134),
 *   - forward pass with per-site rescaling (imputation_hmm.cpp:143-235),
 *   - backward pass and posteriors (imputation_hmm.cpp:237-416),
 *   - monomorphic sites (imputation_hmm.cpp:417-429).
 * rs_impute also returns the chunk log-likelihood sum_l log(AlphaSum_l) of the
 * forward rescaling (no counterpart in the reference).
 *
 * rs_rephase restates the phasing HMM (phase/src/models/phasing_hmm.cpp:65-302) in
 * single precision, its sums over states in the library's fixed order.
 */
#include <math.h>
#include <stdint.h>
#include <stdlib.h>
#include <string.h>

#define DEFINE_IMPUTE(NAME, REAL)                                                                                 \
  static double NAME(int L, const uint8_t* common, const uint8_t* lq, const uint8_t* major, const double* cm,      \
                     const int32_t* comrow, const uint8_t* hvar, int stride, const int64_t* shap_off,            \
                     const int32_t* shap_sites, const uint32_t* states, int K, double nrho, float ed_f, float ee_f,  \
                     const float* HL, const uint8_t* flat, float* HP) {                                          \
    const REAL ed = (REAL)ed_f, ee = (REAL)ee_f;                                                                  \
    uint8_t* poly = (uint8_t*)calloc(L, 1);                                                                       \
    int32_t* plist = (int32_t*)malloc(sizeof(int32_t) * L);                                                       \
    int np = 0;                                                                                                   \
    for (int l = 0; l < L; ++l) poly[l] = common[l];                                                              \
    for (int k = 0; k < K; ++k)                                                                                   \
      for (int64_t j = shap_off[states[k]]; j < shap_off[states[k] + 1]; ++j) poly[shap_sites[j]] = 1;            \
    for (int l = 0; l < L; ++l)                                                                                   \
      if (poly[l]) plist[np++] = l;                                                                               \
    uint8_t* bits = (uint8_t*)malloc((size_t)np * K + 1);                                                         \
    int32_t* lrel = (int32_t*)malloc(sizeof(int32_t) * L);                                                        \
    for (int i = 0; i < np; ++i) lrel[plist[i]] = i;                                                              \
    for (int i = 0; i < np; ++i) {                                                                                \
      const int s = plist[i];                                                                                     \
      for (int k = 0; k < K; ++k) {                                                                               \
        if (common[s]) {                                                                                          \
          const int h = (int)states[k];                                                                           \
          bits[(size_t)i * K + k] = (hvar[(size_t)comrow[s] * stride + (h >> 3)] >> (7 - (h & 7))) & 1;           \
        } else {                                                                                                  \
          bits[(size_t)i * K + k] = major[s];                                                                     \
        }                                                                                                         \
      }                                                                                                           \
    }                                                                                                             \
    for (int k = 0; k < K; ++k)                                                                                   \
      for (int64_t j = shap_off[states[k]]; j < shap_off[states[k] + 1]; ++j) {                                   \
        const int s = shap_sites[j];                                                                              \
        bits[(size_t)lrel[s] * K + k] = !major[s];                                                                \
      }                                                                                                           \
    REAL* t = (REAL*)malloc(sizeof(REAL) * (np + 1));                                                             \
    for (int i = 1; i < np; ++i) {                                                                                \
      double x = -expm1(nrho * (cm[plist[i]] - cm[plist[i - 1]]));                                                \
      x = x < 1e-7 ? 1e-7 : (x > 1.0 - 1e-7 ? 1.0 - 1e-7 : x);                                                    \
      t[i - 1] = (REAL)(float)x;                                                                                  \
    }                                                                                                             \
    REAL* alpha = (REAL*)malloc(sizeof(REAL) * (size_t)np * K + 1);                                               \
    REAL* asum = (REAL*)malloc(sizeof(REAL) * (np + 1));                                                          \
    REAL* beta = (REAL*)malloc(sizeof(REAL) * (K + 1));                                                           \
    double loglik = 0.0;                                                                                          \
    for (int i = 0; i < np; ++i) {                                                                                \
      const int s = plist[i];                                                                                     \
      const int fl = flat[s] || lq[s];                                                                            \
      REAL e[2];                                                                                                  \
      {                                                                                                           \
        const REAL p0 = (REAL)HL[2 * s] * ee + (REAL)HL[2 * s + 1] * ed;                                          \
        const REAL p1 = (REAL)HL[2 * s] * ed + (REAL)HL[2 * s + 1] * ee;                                          \
        e[0] = p0 / (p0 + p1);                                                                                    \
        e[1] = p1 / (p0 + p1);                                                                                    \
      }                                                                                                           \
      REAL sum = 0;                                                                                               \
      REAL* a = alpha + (size_t)i * K;                                                                            \
      if (i == 0) {                                                                                               \
        for (int k = 0; k < K; ++k) {                                                                             \
          a[k] = fl ? (REAL)1 / (REAL)K : e[bits[k]] * ((REAL)1 / (REAL)K);                                        \
          sum += a[k];                                                                                            \
        }                                                                                                         \
        if (fl) sum = 1;                                                                                          \
      } else {                                                                                                    \
        const REAL f1 = t[i - 1] / (REAL)K, f2 = ((REAL)1 - t[i - 1]) / asum[i - 1];                              \
        const REAL* ap = alpha + (size_t)(i - 1) * K;                                                             \
        for (int k = 0; k < K; ++k) {                                                                             \
          a[k] = ap[k] * f2 + f1;                                                                                 \
          if (!fl) a[k] *= e[bits[(size_t)i * K + k]];                                                            \
          sum += a[k];                                                                                            \
        }                                                                                                         \
      }                                                                                                           \
      asum[i] = sum;                                                                                              \
      loglik += log((double)sum);                                                                                 \
    }                                                                                                             \
    REAL bsum_next = 0;                                                                                           \
    for (int i = np - 1; i >= 0; --i) {                                                                           \
      const int s = plist[i];                                                                                     \
      const int fl = flat[s] || lq[s];                                                                            \
      REAL e[2];                                                                                                  \
      {                                                                                                           \
        const REAL p0 = (REAL)HL[2 * s] * ee + (REAL)HL[2 * s + 1] * ed;                                          \
        const REAL p1 = (REAL)HL[2 * s] * ed + (REAL)HL[2 * s + 1] * ee;                                          \
        e[0] = p0 / (p0 + p1);                                                                                    \
        e[1] = p1 / (p0 + p1);                                                                                    \
      }                                                                                                           \
      REAL ph[2] = {0, 0}, bsum = 0;                                                                              \
      const REAL* a = alpha + (size_t)i * K;                                                                      \
      const uint8_t* bi = bits + (size_t)i * K;                                                                   \
      if (i == np - 1) {                                                                                          \
        for (int k = 0; k < K; ++k) {                                                                             \
          ph[bi[k]] += a[k];                                                                                      \
          beta[k] = fl ? (REAL)1 / (REAL)K : e[bi[k]] * ((REAL)1 / (REAL)K);                                        \
          bsum += beta[k];                                                                                        \
        }                                                                                                         \
        if (fl) bsum = 1;                                                                                         \
      } else {                                                                                                    \
        const REAL f1 = t[i] / (REAL)K, f2 = ((REAL)1 - t[i]) / bsum_next;                                        \
        for (int k = 0; k < K; ++k) {                                                                             \
          const REAL pc = beta[k] * f2 + f1;                                                                      \
          ph[bi[k]] += a[k] * pc;                                                                                 \
          beta[k] = fl ? pc : pc * e[bi[k]];                                                                      \
          bsum += beta[k];                                                                                        \
        }                                                                                                         \
      }                                                                                                           \
      REAL po0, po1;                                                                                              \
      if (fl) {                                                                                                   \
        po0 = ph[0] * ee + ph[1] * ed;                                                                            \
        po1 = ph[0] * ed + ph[1] * ee;                                                                            \
        if (!flat[s]) {                                                                                           \
          po0 *= (REAL)HL[2 * s];                                                                                 \
          po1 *= (REAL)HL[2 * s + 1];                                                                             \
        }                                                                                                         \
      } else {                                                                                                    \
        const REAL h0 = ph[0] / e[0], h1 = ph[1] / e[1];                                                          \
        po0 = (h0 * ee + h1 * ed) * (REAL)HL[2 * s];                                                              \
        po1 = (h0 * ed + h1 * ee) * (REAL)HL[2 * s + 1];                                                          \
      }                                                                                                           \
      HP[2 * s] = (float)(po0 / (po0 + po1));                                                                     \
      HP[2 * s + 1] = (float)(po1 / (po0 + po1));                                                                 \
      bsum_next = bsum;                                                                                           \
    }                                                                                                             \
    for (int l = 0; l < L; ++l) {                                                                                 \
      if (poly[l]) continue;                                                                                      \
      REAL p0 = major[l] ? ed : ee, p1 = major[l] ? ee : ed;                                                      \
      if (!flat[l]) {                                                                                             \
        p0 *= (REAL)HL[2 * l];                                                                                    \
        p1 *= (REAL)HL[2 * l + 1];                                                                                \
      }                                                                                                           \
      HP[2 * l] = (float)(p0 / (p0 + p1));                                                                        \
      HP[2 * l + 1] = (float)(p1 / (p0 + p1));                                                                    \
    }                                                                                                             \
    free(poly); free(plist); free(bits); free(lrel); free(t); free(alpha); free(asum); free(beta);                \
    return loglik;                                                                                                \
  }

DEFINE_IMPUTE(impute_f64, double)
DEFINE_IMPUTE(impute_f32, float)

/* HP for one haplotype with conditioning set `states` (sorted reference ids).
 * precision: 64 or 32. Returns the chunk log-likelihood. */
double rs_impute(int precision, int L, const uint8_t* common, const uint8_t* lq, const uint8_t* major,
                 const double* cm, const int32_t* comrow, const uint8_t* hvar, int stride, const int64_t* shap_off,
                 const int32_t* shap_sites, const uint32_t* states, int K, double nrho, float ed, float ee,
                 const float* HL, const uint8_t* flat, float* HP) {
  if (precision == 64)
    return impute_f64(L, common, lq, major, cm, comrow, hvar, stride, shap_off, shap_sites, states, K, nrho, ed, ee,
                      HL, flat, HP);
  return impute_f32(L, common, lq, major, cm, comrow, hvar, stride, shap_off, shap_sites, states, K, nrho, ed, ee, HL,
                    flat, HP);
}

/* Per-window state posteriors, FP64: the label HMM of the learned state
 * selection (no counterpart in the reference). For the conditioning set built
 * as above, mass[w * K + k] = sum over the polymorphic sites l with
 * site_win[l] == w of alpha_l(k) beta_l(k) / sum_k' alpha_l(k') beta_l(k'),
 * alpha_l including the emission at l and beta_l the backward message
 * without it (beta = 1 at the last site); nsites[w] counts those sites. */
void rs_state_post(int L, const uint8_t* common, const uint8_t* lq, const uint8_t* major, const double* cm,
                   const int32_t* comrow, const uint8_t* hvar, int stride, const int64_t* shap_off,
                   const int32_t* shap_sites, const uint32_t* states, int K, double nrho, float ed_f, float ee_f,
                   const float* HL, const uint8_t* flat, const int32_t* site_win, int nwin, double* mass,
                   int32_t* nsites) {
  const double ed = ed_f, ee = ee_f;
  uint8_t* poly = (uint8_t*)calloc(L, 1);
  int32_t* plist = (int32_t*)malloc(sizeof(int32_t) * L);
  int np = 0;
  for (int l = 0; l < L; ++l) poly[l] = common[l];
  for (int k = 0; k < K; ++k)
    for (int64_t j = shap_off[states[k]]; j < shap_off[states[k] + 1]; ++j) poly[shap_sites[j]] = 1;
  for (int l = 0; l < L; ++l)
    if (poly[l]) plist[np++] = l;
  uint8_t* bits = (uint8_t*)malloc((size_t)np * K + 1);
  int32_t* lrel = (int32_t*)malloc(sizeof(int32_t) * L);
  for (int i = 0; i < np; ++i) lrel[plist[i]] = i;
  for (int i = 0; i < np; ++i) {
    const int s = plist[i];
    for (int k = 0; k < K; ++k) {
      const int h = (int)states[k];
      bits[(size_t)i * K + k] =
          common[s] ? (hvar[(size_t)comrow[s] * stride + (h >> 3)] >> (7 - (h & 7))) & 1 : major[s];
    }
  }
  for (int k = 0; k < K; ++k)
    for (int64_t j = shap_off[states[k]]; j < shap_off[states[k] + 1]; ++j)
      bits[(size_t)lrel[shap_sites[j]] * K + k] = !major[shap_sites[j]];
  double* t = (double*)malloc(sizeof(double) * (np + 1));
  for (int i = 1; i < np; ++i) {
    double x = -expm1(nrho * (cm[plist[i]] - cm[plist[i - 1]]));
    x = x < 1e-7 ? 1e-7 : (x > 1.0 - 1e-7 ? 1.0 - 1e-7 : x);
    t[i - 1] = (double)(float)x;
  }
  double* alpha = (double*)malloc(sizeof(double) * (size_t)np * K + 8);
  double* beta = (double*)malloc(sizeof(double) * (K + 1));
  double* nb = (double*)malloc(sizeof(double) * (K + 1));
  double* em = (double*)malloc(sizeof(double) * 2 * (np + 1));
  for (int i = 0; i < np; ++i) {
    const int s = plist[i];
    if (flat[s] || lq[s]) {
      em[2 * i] = em[2 * i + 1] = 1.0;
    } else {
      const double p0 = (double)HL[2 * s] * ee + (double)HL[2 * s + 1] * ed;
      const double p1 = (double)HL[2 * s] * ed + (double)HL[2 * s + 1] * ee;
      em[2 * i] = p0 / (p0 + p1);
      em[2 * i + 1] = p1 / (p0 + p1);
    }
  }
  for (int i = 0; i < np; ++i) {
    double* a = alpha + (size_t)i * K;
    double sum = 0;
    for (int k = 0; k < K; ++k) {
      const double prev = i == 0 ? 1.0 / K : alpha[(size_t)(i - 1) * K + k] * (1.0 - t[i - 1]) + t[i - 1] / K;
      a[k] = prev * em[2 * i + bits[(size_t)i * K + k]];
      sum += a[k];
    }
    for (int k = 0; k < K; ++k) a[k] /= sum;
  }
  for (int w = 0; w < nwin; ++w) nsites[w] = 0;
  for (size_t j = 0; j < (size_t)nwin * K; ++j) mass[j] = 0.0;
  for (int k = 0; k < K; ++k) beta[k] = 1.0;
  for (int i = np - 1; i >= 0; --i) {
    if (i < np - 1) {
      double se = 0;
      for (int k = 0; k < K; ++k) {
        nb[k] = em[2 * (i + 1) + bits[(size_t)(i + 1) * K + k]] * beta[k];
        se += nb[k];
      }
      for (int k = 0; k < K; ++k) beta[k] = nb[k] / se * (1.0 - t[i]) + t[i] / K;
    }
    const double* a = alpha + (size_t)i * K;
    double z = 0;
    for (int k = 0; k < K; ++k) z += a[k] * beta[k];
    const int w = site_win[plist[i]];
    nsites[w]++;
    for (int k = 0; k < K; ++k) mass[(size_t)w * K + k] += a[k] * beta[k] / z;
  }
  free(poly); free(plist); free(bits); free(lrel); free(t); free(alpha); free(beta); free(nb); free(em);
}

/* The sum of K values in the library's order: state k belongs to lane k % 32 of
 * warp (k / 32) % 8, which adds its states in increasing order; lanes pairwise at
 * distances 16, 8, 4, 2, 1, then warps at 1, 2, 4. add[i] of 256 start at 0. */
static float tree256(const float* lanes) {
  float a[256];
  memcpy(a, lanes, sizeof a);
  for (int o = 16; o > 0; o >>= 1)
    for (int w = 0; w < 8; ++w)
      for (int l = 0; l < o; ++l) a[32 * w + l] += a[32 * w + l + o];
  for (int o = 1; o < 8; o <<= 1)
    for (int w = 0; w < 8; w += 2 * o) a[32 * w] += a[32 * (w + o)];
  return a[0];
}

static float hadd8(const float* v) {
  return ((v[0] + v[4]) + (v[1] + v[5])) + ((v[2] + v[6]) + (v[3] + v[7]));
}

enum { T_HOM = 3, T_FLAT = 4 };
typedef struct { int site, typ, alt, seg, miss; } var_t;

static float trans(const double* cm, int a, int b, double nrho) {
  double x = -expm1(nrho * (cm[b] - cm[a]));
  x = x < 1e-7 ? 1e-7 : (x > 1.0 - 1e-7 ? 1.0 - 1e-7 : x);
  return (float)x;
}

/* One pass (dir 1 forward, -1 backward) over the nv VAR sites; the messages of the
 * entries wanted by the other pass go to srow / ssum / stot (segment ends forward,
 * segment starts backward) and mrow / msum (flat hets). */
static void phase_pass(int dir, int K, int nv, const var_t* v, const int* start, const double* cm, double nrho, float ed,
                       float ee, const uint8_t* bits, float* srow, float* ssum, float* stot, float* mrow, float* msum) {
  float* prob = (float*)calloc((size_t)K * 8, sizeof(float));
  float sumH[8], sumT = 1.0f;
  const float mism = ed / ee;
  for (int s = 0; s < nv; ++s) {
    const int i = dir > 0 ? s : nv - 1 - s;
    const var_t* e = v + i;
    const int first = i == start[e->seg], last = i == start[e->seg + 1] - 1;
    if (s == 0 && e->typ == T_FLAT) {
      for (int j = 0; j < 8 * K; ++j) prob[j] = 1.0f / (float)(8u * (unsigned)K);
      for (int h = 0; h < 8; ++h) sumH[h] = 0.125f;
    } else {
      float tF[8], ntp = 0.f, part[8][256];
      memset(part, 0, sizeof part);
      if (s > 0) {
        const float yt = trans(cm, v[dir > 0 ? i - 1 : i].site, v[dir > 0 ? i : i + 1].site, nrho);
        const float sc = yt / ((float)K * sumT);
        for (int h = 0; h < 8; ++h) tF[h] = sumH[h] * sc;
        ntp = (1.0f - yt) / sumT;
      }
      const int collapse = s > 0 && (dir > 0 ? first : last);
      for (int k = 0; k < K; ++k) {
        float* p = prob + (size_t)k * 8;
        const int a = bits[(size_t)i * K + k];
        const float all = collapse ? hadd8(p) : 0.f;
        for (int h = 0; h < 8; ++h) {
          float em = 1.0f;
          if (e->typ < 3) em = a == (((7 - h) >> (2 - e->typ)) & 1) ? ee : ed;
          else if (e->typ == T_HOM) em = a != e->alt ? mism : 1.0f;
          p[h] = s == 0 ? em : fmaf(collapse ? all : p[h], ntp, tF[h]) * em;
          part[h][k & 255] += p[h];
        }
      }
      for (int h = 0; h < 8; ++h) sumH[h] = tree256(part[h]);
      sumT = hadd8(sumH);
    }
    if (dir > 0 ? last : first) {
      memcpy(srow + (size_t)e->seg * K * 8, prob, sizeof(float) * 8 * K);
      memcpy(ssum + e->seg * 8, sumH, sizeof sumH);
      stot[e->seg] = sumT;
    }
    if (e->typ == T_FLAT) {
      memcpy(mrow + (size_t)e->miss * K * 8, prob, sizeof(float) * 8 * K);
      memcpy(msum + e->miss * 8, sumH, sizeof sumH);
    }
  }
  free(prob);
}

/* phasing_hmm::rephaseHaplotypes on one target; u[w] is word w of its random stream
 * as a float in [0, 1). h0 and h1 are rewritten. Returns nonzero when a diplotype
 * draw saw an invalid sum (the reference asserts there, phasing_hmm.cpp:175). */
int rs_rephase(int L, const uint8_t* common, const uint8_t* lq, const uint8_t* major, const double* cm,
               const int32_t* comrow, const uint8_t* hvar, int stride, const int64_t* shap_off,
               const int32_t* shap_sites, const uint32_t* states, int K, double nrho, float ed, float ee,
               const uint8_t* flat, const float* u, uint8_t* h0, uint8_t* h1) {
  uint8_t* poly = (uint8_t*)malloc(L);
  memcpy(poly, common, L);
  for (int k = 0; k < K; ++k)
    for (int64_t j = shap_off[states[k]]; j < shap_off[states[k] + 1]; ++j) poly[shap_sites[j]] = 1;
  var_t* v = (var_t*)malloc(sizeof(var_t) * (L + 1));
  int* start = (int*)malloc(sizeof(int) * (L + 2));
  int32_t* at = (int32_t*)malloc(sizeof(int32_t) * L);
  int nv = 0, nhet = 0, nmiss = 0;
  for (int l = 0; l < L; ++l) {
    at[l] = -1;
    if (!poly[l]) continue;
    const int peak = !flat[l] && !lq[l], het = h0[l] != h1[l];
    if (!peak && !het) continue;
    var_t e = {l, T_HOM, h0[l], (nhet > 0 ? nhet - 1 : 0) / 3, -1};
    if (peak && het) {
      e.typ = nhet % 3;
      e.seg = nhet / 3;
      if (nhet > 0 && e.typ == 0) start[e.seg] = nv;
      ++nhet;
    } else if (!peak) {
      e.typ = T_FLAT;
      e.miss = nmiss++;
    }
    at[l] = nv;
    v[nv++] = e;
  }
  const int nseg = (nhet > 0 ? nhet - 1 : 0) / 3 + 1;
  start[0] = 0;
  start[nseg] = nv;
  uint8_t* bits = (uint8_t*)malloc((size_t)nv * K + 1);
  for (int i = 0; i < nv; ++i)
    for (int k = 0; k < K; ++k) {
      const int s = v[i].site, h = (int)states[k];
      bits[(size_t)i * K + k] =
          common[s] ? (hvar[(size_t)comrow[s] * stride + (h >> 3)] >> (7 - (h & 7))) & 1 : major[s];
    }
  for (int k = 0; k < K; ++k)
    for (int64_t j = shap_off[states[k]]; j < shap_off[states[k] + 1]; ++j)
      if (at[shap_sites[j]] >= 0) bits[(size_t)at[shap_sites[j]] * K + k] = !major[shap_sites[j]];
  const size_t row = sizeof(float) * 8 * K;
  float *sr[2], *ss[2], *st[2], *mr[2], *ms[2];
  for (int d = 0; d < 2; ++d) {  /* 0 forward, 1 backward */
    sr[d] = (float*)malloc(row * nseg);
    ss[d] = (float*)calloc(8 * (size_t)nseg, sizeof(float));
    st[d] = (float*)calloc((size_t)nseg, sizeof(float));
    mr[d] = (float*)malloc(row * (nmiss + 1));
    ms[d] = (float*)malloc(sizeof(float) * 8 * (nmiss + 1));
    phase_pass(d ? -1 : 1, K, nv, v, start, cm, nrho, ed, ee, bits, sr[d], ss[d], st[d], mr[d], ms[d]);
  }
  int* dip = (int*)malloc(sizeof(int) * nseg);
  int bad = 0;
  dip[0] = 7;
  for (int g = 0; nv > 0 && g < nseg; ++g) {
    float dp[8], sd = 0.f;
    int wrong = 0;
    if (g == 0) {
      for (int d = 0; d < 8; ++d) dp[d] = (ss[1][d] / st[1][0]) * (ss[1][7 - d] / st[1][0]);
    } else {
      /* TRANS_HAP between the segments g - 1 and g */
      const int b = g - 1, prev = dip[b], end = start[g] - 1;
      const float yt = trans(cm, v[end].site, v[end + 1].site, nrho);
      const float fact2 = (1.0f - yt) / st[0][b];
      float hp[64], sum = 0.f;
      for (int x = 0; x < 8; ++x) {
        const float fact1 = (ss[0][b * 8 + x] / st[0][b]) * yt / (float)K;
        for (int y = 0; y < 8; ++y) {
          float part[256] = {0};
          for (int k = 0; k < K; ++k)
            part[k & 255] = fmaf(fmaf(sr[0][((size_t)b * K + k) * 8 + x], fact2, fact1),
                                 sr[1][((size_t)g * K + k) * 8 + y], part[k & 255]);
          hp[8 * x + y] = tree256(part);
        }
        sum += hadd8(hp + 8 * x);
      }
      for (int d = 0; d < 8; ++d) dp[d] = (hp[prev * 8 + d] / sum) * (hp[(7 - prev) * 8 + (7 - d)] / sum);
      wrong = !(sum >= 1.17549435e-38f) || isinf(sum);
    }
    for (int d = 0; d < 8; ++d) sd += dp[d];
    if (g > 0) wrong |= !(sd >= 1.17549435e-38f) || isinf(sd);
    const float w = u[g] * sd;
    float cs = dp[0];
    dip[g] = 7;
    for (int d = 0; d < 7; ++d) {
      if (w <= cs) {
        dip[g] = d;
        break;
      }
      cs += dp[d + 1];
    }
    if (wrong) dip[g] = dip[g - 1];
    bad |= wrong;
  }
  int mono = 0;
  for (int l = 0; l < L; ++l)
    if (!poly[l] && h0[l] != h1[l]) {  /* hets at monomorphic sites (phasing_hmm.cpp:293-301) */
      h0[l] = u[nseg + nmiss + mono++] < 0.5f;
      h1[l] = !h0[l];
    }
  for (int i = 0; i < nv; ++i) {
    const var_t* e = v + i;
    const int a = dip[e->seg], b = 7 - a;
    if (e->typ < 3) {
      h0[e->site] = ((7 - a) >> (2 - e->typ)) & 1;
      h1[e->site] = ((7 - b) >> (2 - e->typ)) & 1;
    } else if (e->typ == T_FLAT) {
      /* IMPUTE_FLAT_HET (phasing_hmm.h:414-447) */
      float of[2];
      for (int x = 0; x < 2; ++x) {
        const int h = x ? b : a;
        const float sR = 1.0f / ms[1][e->miss * 8 + h], sL = 1.0f / ms[0][e->miss * 8 + h];
        float part[2][256] = {{0}};
        for (int k = 0; k < K; ++k) {
          float* q = &part[bits[(size_t)i * K + k]][k & 255];
          *q = fmaf(mr[1][((size_t)e->miss * K + k) * 8 + h] * sR, mr[0][((size_t)e->miss * K + k) * 8 + h] * sL, *q);
        }
        const float t0 = tree256(part[0]), t1 = tree256(part[1]);
        of[x] = fmaxf(0.0f, fminf(1.0f, t1 / (t0 + t1)));
      }
      float p01 = fmaf(1.0f - of[0], ee, of[0] * ed) * fmaf(of[1], ee, (1.0f - of[1]) * ed);
      float p10 = fmaf(of[0], ee, (1.0f - of[0]) * ed) * fmaf(1.0f - of[1], ee, of[1] * ed);
      const float sum = p01 + p10;
      p01 = fminf(fmaxf(p01 / sum, 0.0f), 1.0f);
      p10 = fminf(fmaxf(p10 / sum, 0.0f), 1.0f);
      h0[e->site] = !((double)u[nseg + e->miss] * (double)(p01 + p10) < (double)p01);
    }
  }
  for (int d = 0; d < 2; ++d) {
    free(sr[d]); free(ss[d]); free(st[d]); free(mr[d]); free(ms[d]);
  }
  free(poly); free(v); free(start); free(at); free(bits); free(dip);
  return bad;
}

/*
 * count_common.cuh -- device code shared by the counting kernels: the
 * weights' fixed-point products and the reference's FP64 binning of one
 * pair.  Included by count.cu and by the count32_*.cu translation units.
 */
#ifndef FCFCG_COUNT_COMMON_CUH
#define FCFCG_COUNT_COMMON_CUH
#include <cuda_runtime.h>
#include <float.h>
#include <stdint.h>
#include <string.h>

#include "fcfcg_internal.h"

/* Kernel binning codes: the public FCFCG_BIN_* (0 iso, 1 (s,mu), 2
 * (s_perp,pi)), their edges from tables; iso (3) and (s,mu) (4) with evenly
 * spaced s edges, (s_perp,pi) (5) with evenly spaced pi edges, which come
 * from the value itself; and (6) every pair in FP64, the launch's binning. */
#define BIN_ISOLIN 3
#define BIN_SMULIN 4
#define BIN_SPILIN 5
#define BIN_F64 6
#define IS_SPI(B) ((B) == FCFCG_BIN_SPI || (B) == BIN_SPILIN)
#define IS_ISO(B) ((B) == FCFCG_BIN_ISO || (B) == BIN_ISOLIN)
#define IS_SMU(B) ((B) == FCFCG_BIN_SMU || (B) == BIN_SMULIN)
#define LINS(B) ((B) == BIN_ISOLIN || (B) == BIN_SMULIN)
#define LINP(B) ((B) == BIN_SPILIN)
/* survey (s_perp, pi): the line-of-sight prefilter */
#define LOSCUT(G, B) ((G) == FCFCG_GEOM_SURVEY && IS_SPI(B))

#define FULLMASK 0xffffffffu

/* ------------------------------------------------------------------------ */
/* Accumulators.                                                            */

/* Add a signed 64-bit value to a 128-bit two's complement accumulator. */
__device__ __forceinline__ void add128(unsigned long long *lohi, long long v) {
  unsigned long long u = (unsigned long long) v;
  unsigned long long old = atomicAdd(lohi, u);
  unsigned long long hi = ((old + u) < old ? 1ull : 0ull) +
                          (v < 0 ? ~0ull : 0ull);
  if (hi) atomicAdd(lohi + 1, hi);
}

/*
 * Fixed-point product of two weights scaled to |w| <= 1, with F = 51
 * fractional bits (FCFCG_FIX_F).  A weight is held as an integer part
 * wi = round(w 2^30) and a float remainder wr = w - wi 2^-30 (|wr| <= 2^-31):
 *   w_a w_b 2^51 = wi_a wi_b 2^-9 + (w_a wr_b + wr_a w_b) 2^51 (+ wr wr).
 * The first term is an exact 64-bit product rounded by a shift; the cross
 * term (|.| <= 2^21) is rounded with the 1.5 * 2^23 float trick; wr wr
 * (<= 2^-11 of a unit) is dropped.  No 64-bit float conversions.  The
 * function is symmetric in a and b (two rounded products and a commutative
 * sum, no fused multiply-add), and every path uses it, so a pair adds the
 * same integer whichever point is A's: weighted sums do not depend
 * on the order of the points within a cell.
 */
__device__ __forceinline__ long long fix_prod(int ia, float ra, float fa,
    int ib, float rb, float fb) {
  const long long p = (long long) ia * (long long) ib;
  const long long main = (p + (1ll << 8)) >> 9;
  const float c = __fadd_rn(__fmul_rn(fa, rb), __fmul_rn(ra, fb));
  const float t = __fmaf_rn(c, 2251799813685248.0f /* 2^51 */, 12582912.0f);
  return main + (long long) (__float_as_int(t) - 0x4B400000);
}

__device__ __forceinline__ long long fix_prod_pair(const fcfcg_launch &L,
    uint32_t a, uint32_t b) {
  const int2 wa = ((const int2 *) L.A.wq)[a];
  const int2 wb = ((const int2 *) L.B.wq)[b];
  const float fa = ((const float4 *) L.A.l4)[a].w;
  const float fb = ((const float4 *) L.B.l4)[b].w;
  return fix_prod(wa.x, __int_as_float(wa.y), fa, wb.x, __int_as_float(wb.y),
                  fb);
}

/* ------------------------------------------------------------------------ */
/* FP64 binning of one pair, exactly as the reference's scalar FP64 code.   */

__device__ __forceinline__ int ref_lookup(const uint16_t *__restrict__ tab,
    long off, long ntab, int num, const double *__restrict__ edge, double v) {
  long t = (long) __double2int_rz(v) - off;
  if (!(v == v) || t < 0 || t >= ntab) return -1;   /* never indexes outside */
  int idx = __ldg(tab + t);
  if (idx >= num) {                 /* hybrid entry: walk down */
    idx -= num;
    while (idx != 0 && v < __ldg(edge + idx)) idx--;
  }
  return idx;
}

/* floor(sqrt(p)) of 0 <= p <= 255^2, what the reference's mutab holds
 * (setup_cf.c:513-531). */
__device__ __forceinline__ int ref_isqrt(int p) {
  int k = (int) sqrtf((float) p);
  while (k * k > p) k--;
  while ((k + 1) * (k + 1) <= p) k++;
  return k;
}

/*
 * mu bin of mu^2 = num / den (survey: LOS, fl(num / m2) / den): the
 * reference's mutab[(int) fl(mu^2 nmu^2)], i.e. k with k^2 <= that product <
 * (k + 1)^2; -1: mu >= 1, dropped.  FP32 decides where it can: q = nmu
 * sqrt(num) / sqrt(den) is within 4.3e-7 q of the exact value (conversions
 * 2^-25 of the root each, sqrt.approx 2^-23, rsqrt.approx 2^-22.9, products
 * 2^-24 each; LOS 6.4e-7 q) and the reference's roundings are far below, so
 * a q farther than twice that and 1e-6 from an integer has its bin; the
 * others take the FP64 divisions (a dozen operations each, of a pipe of 2
 * lanes per SM).
 */
template <bool LOS>
__device__ __forceinline__ int ref_mu(const fcfcg_launch &L, double num,
    double m2, double den) {
  const float nf = (float) num, df = (float) den, mf = (float) m2;
  float q, rd;
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(q) : "f"(nf));
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(rd) : "f"(df));
  if (LOS) {
    float rm;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(rm) : "f"(mf));
    q *= rm;
  }
  q = (float) L.nmu * q * rd;
  const int k = (int) q;
  const float f = q - (float) k, tol = fmaf(q, LOS ? 1.3e-6f : 9.6e-7f, 1e-6f);
  if (df > 1e-15f && nf > 1e-30f && (!LOS || mf > 1e-15f) && f > tol &&
      f < 1.f - tol && k < L.nmu)
    return k;
  const int nmu2 = L.nmu * L.nmu;
  if (LOS) num = __ddiv_rn(num, m2);
  int p = (den < DBL_EPSILON) ? 0
          : __double2int_rz(__dmul_rn(__ddiv_rn(num, den), (double) nmu2));
  if (p < 0) return -1;
  if (p >= nmu2) {
    if (!L.mu_one) return -1;
    p = nmu2 - 1;
  }
  return ref_isqrt(p);
}

/* Periodic box, src/fcfc/2pt_box/metric_common.c:140-235.
 * (dx, dy, dz) = (x1 + shift) - x2 already formed. */
static __device__ int ref_bin_box(const fcfcg_launch &L, double dx, double dy,
    double dz) {
  if (L.bintype == FCFCG_BIN_SPI) {
    double pi = fabs(dz);
    if (pi >= L.pmax) return -1;
    if (!L.pmin0 && pi < L.pmin) return -1;
    double d = __dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy));
    if (d >= L.s2max) return -1;
    if (!L.smin0 && d < L.s2min) return -1;
    int si = ref_lookup(L.rs, L.rsoff, L.nrs, L.ns, L.s2edge, d);
    int pi_ = ref_lookup(L.rp, L.rpoff, L.nrp, L.np, L.pedge, pi);
    if (si < 0 || pi_ < 0) return -1;
    return si + pi_ * L.ns;
  }
  double dz2 = __dmul_rn(dz, dz);
  double d = __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), dz2);
  if (d >= L.s2max) return -1;
  if (!L.smin0 && d < L.s2min) return -1;
  int mi = 0;
  if (L.bintype == FCFCG_BIN_SMU) {
    mi = ref_mu<false>(L, dz2, 1.0, d);
    if (mi < 0) return -1;
  }
  int si = ref_lookup(L.rs, L.rsoff, L.nrs, L.ns, L.s2edge, d);
  if (si < 0) return -1;
  return si + mi * L.ns;
}

/* Survey, src/fcfc/2pt/metric_common.c:142-260. */
static __device__ int ref_bin_survey(const fcfcg_launch &L, double x1, double y1,
    double z1, double s1, double x2, double y2, double z2, double s2) {
  if (L.bintype == FCFCG_BIN_ISO) {
    double dx = __dsub_rn(x1, x2), dy = __dsub_rn(y1, y2),
           dz = __dsub_rn(z1, z2);
    double d = __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)),
                         __dmul_rn(dz, dz));
    if (d >= L.s2max) return -1;
    if (!L.smin0 && d < L.s2min) return -1;
    return ref_lookup(L.rs, L.rsoff, L.nrs, L.ns, L.s2edge, d);
  }
  double t = __dmul_rn(__dadd_rn(__dadd_rn(__dmul_rn(x1, x2),
                                           __dmul_rn(y1, y2)),
                                 __dmul_rn(z1, z2)), 2.0);
  double s = __dadd_rn(s1, s2);
  if (L.bintype == FCFCG_BIN_SMU) {
    double d = __dsub_rn(s, t);
    if (d >= L.s2max) return -1;
    if (!L.smin0 && d < L.s2min) return -1;
    const double dd = __dsub_rn(s1, s2);
    const int k = ref_mu<true>(L, __dmul_rn(dd, dd), __dadd_rn(s, t), d);
    if (k < 0) return -1;
    int si = ref_lookup(L.rs, L.rsoff, L.nrs, L.ns, L.s2edge, d);
    if (si < 0) return -1;
    return si + k * L.ns;
  }
  double dd = __dsub_rn(s1, s2);
  double pi2 = __ddiv_rn(__dmul_rn(dd, dd), __dadd_rn(s, t));
  if (pi2 >= L.pmax) return -1;
  if (!L.pmin0 && pi2 < L.pmin) return -1;
  double d = __dsub_rn(__dsub_rn(s, t), pi2);
  if (d >= L.s2max) return -1;
  if (!L.smin0 && d < L.s2min) return -1;
  if (d < 0) d = 0;      /* (int) of a value in (-1, 0) is 0 */
  int si = ref_lookup(L.rs, L.rsoff, L.nrs, L.ns, L.s2edge, d);
  int pi_ = ref_lookup(L.rp, L.rpoff, L.nrp, L.np, L.pedge, pi2);
  if (si < 0 || pi_ < 0) return -1;
  return si + pi_ * L.ns;
}

/* Exact bin of sorted point a (catalogue A) and b (catalogue B) with the
 * image code of the cell pair (box).  The image shift goes to the A point,
 * or for auto counts to the point with the smaller input index. */
static __device__ int ref_bin_pair(const fcfcg_launch &L, uint32_t a, uint32_t b,
    uint32_t code, const double *box) {
  if (L.geometry == FCFCG_GEOM_SURVEY)
    return ref_bin_survey(L, L.A.x[a], L.A.y[a], L.A.z[a], L.A.s[a],
                          L.B.x[b], L.B.y[b], L.B.z[b], L.B.s[b]);
  const int wx = (int) (code & 3u) - 1, wy = (int) ((code >> 2) & 3u) - 1,
            wz = (int) ((code >> 4) & 3u) - 1;
  const double shx = -wx * box[0], shy = -wy * box[1],
               shz = -wz * box[2];
  const double xa = L.A.x[a], ya = L.A.y[a], za = L.A.z[a];
  const double xb = L.B.x[b], yb = L.B.y[b], zb = L.B.z[b];
  double dx, dy, dz;
  if (code == 21u) {
    /* no image shift: the order changes the signs alone */
    dx = __dsub_rn(xa, xb);
    dy = __dsub_rn(ya, yb);
    dz = __dsub_rn(za, zb);
  } else if (!L.isauto || L.A.id[a] < L.B.id[b]) {
    dx = __dsub_rn(__dadd_rn(xa, shx), xb);
    dy = __dsub_rn(__dadd_rn(ya, shy), yb);
    dz = __dsub_rn(__dadd_rn(za, shz), zb);
  } else {
    dx = __dsub_rn(__dsub_rn(xb, shx), xa);
    dy = __dsub_rn(__dsub_rn(yb, shy), ya);
    dz = __dsub_rn(__dsub_rn(zb, shz), za);
  }
  return ref_bin_box(L, dx, dy, dz);
}

/* Adjoint: FP64 gradient contributions of one pair with a known bin. */
__device__ __forceinline__ void adj_pair(const fcfcg_launch &L, uint32_t a,
    uint32_t b, int bin) {
  const double g = __ldg(L.gadj + bin);
  atomicAdd(L.dA + a, __dmul_rn(L.B.w[b], g));
  atomicAdd(L.dB + b, __dmul_rn(L.A.w[a], g));
}

#define CT32_THREADS 256
typedef void (*kfun_t)(const fcfcg_launch);

/* The tile kernel's instantiations, one family per translation unit
 * (count32_box.cu, count32_survey.cu, count32_batch.cu, count32_adj.cu,
 * count32_f64.cu): the kernel for a binning code and weighting, or NULL. */
kfun_t fcfcg_pick32_box(int bin, int wt);
kfun_t fcfcg_pick32_survey(int bin, int wt);
kfun_t fcfcg_pick32_batch(int bin, int wt);
kfun_t fcfcg_pick32_adj(int geom, int bin);
kfun_t fcfcg_pick64(int geom, int wt, int adj);

#endif

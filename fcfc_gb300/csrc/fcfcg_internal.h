/*
 * fcfcg_internal.h -- structures shared by the C host layer and the CUDA
 * kernels of the pair-counting engine.  Plain C, no CUDA types.
 */
#ifndef FCFCG_INTERNAL_H
#define FCFCG_INTERNAL_H

#include <stddef.h>
#include <stdint.h>

#include "../../include/fcfcg.h"

#ifdef __cplusplus
extern "C" {
#endif

#define FCFCG_MAX_SLOT 8
#define FCFCG_MAX_STENCIL 4096
#define FCFCG_FIX_F 51            /* fractional bits of a weight product */
/* FP32 edge-window tables (of which only the cells per octave are used, for
 * fcfcg_bins_info): one uint16 per cell of width w = 2^-shift units of the
 * binned quantity; cell i covers [i w, (i + 1) w). */
#define FCFCG_FTAB_BIN_MASK 0x0FFFu /* bin at the cell start, or "out" */
#define FCFCG_FTAB_LO 0x1000u     /* an edge lies in [i w - w/2, i w] */
#define FCFCG_FTAB_HI 0x2000u     /* an edge lies in [(i+1) w, (i+1) w + w/2] */
#define FCFCG_FTAB_CX1 0x4000u    /* exactly one edge strictly inside */
#define FCFCG_FTAB_CXM 0x8000u    /* several edges strictly inside */
#define FCFCG_FTAB_MAXBIN 4094    /* largest bin index an FP32 table holds */
#define FCFCG_FTAB_MAXLEN 4096    /* cells of an FP32 table */

/* An edge table (host): n cells of the value's FP32 bits >> lg, from cell off
 * on, (edge, 1.5 2^23 + column) each, then two entries for the values below: no
 * edge near, and ambiguous.  For windows below margin of a cell; cut: there are
 * edges below the cells; amb: the ambiguous share of the range.  No table: n =
 * 0. */
#define FCFCG_NETAB 3
typedef struct {
  float *t;
  int n, lg, cut;
  long off;
  double margin, amb;
} fcfcg_etab;

/*
 * One binned quantity (s^2, s_perp^2, pi or pi^2), as FCFC looks it up:
 * reference table rtab over (int) v - roff with FCFC's integer / hybrid
 * semantics, and the FP32 edge-window table ftab over (int) v - foff.
 */
typedef struct {
  int nbin;
  int tabtype;
  double *edge;          /* nbin + 1 rescaled edges (host) */
  uint16_t *rtab;        /* reference table (host) */
  long nrtab, roff;
  uint16_t *ftab;        /* FP32 window table (host) */
  long nftab, foff;      /* cells, index of the first cell */
  int fshift;            /* cell width 2^fshift units */
  int flog;              /* > 0: cells are the FP32 bit pattern >> flog
                            (2^(23 - flog) cells per octave), for bins
                            that are not linear; 0: uniform cells */
  float *fedge;          /* nbin + 1 edges rounded to FP32 (host) */
  double vmin, vmax;     /* edge[0], edge[nbin] */
  int min0;              /* edge[0] == 0: no lower range check (smin0) */
  /* edge tables of the tile kernel: the general one and, where edges are too
   * close for it, finer ones with margins of a half and an eighth of a cell
   * (bins.c:fcfcg_axis_etab) */
  fcfcg_etab etab[FCFCG_NETAB];
} fcfcg_axis;

typedef struct {
  int geometry, bintype;
  int ns, nmu, np;
  long ntot;
  double rescale;
  double box[3];         /* rescaled */
  double box_raw[3];     /* as configured */
  double *sbin_raw, *pbin_raw;
  fcfcg_axis s;          /* s^2 (or s_perp^2) */
  fcfcg_axis p;          /* pi (box) or pi^2 (survey) */
  int mu_one;            /* mu = 1 in the last mu bin (WITH_MU_ONE) */
} fcfcg_bins;

int fcfcg_bins_setup(const fcfcg_binning *cfg, fcfcg_bins *b, char *err,
    size_t errlen);
void fcfcg_bins_release(fcfcg_bins *b);
/* Build the FP32 window table of an axis (ftab / foff / nftab); allow_log:
 * a bit-pattern table may replace a uniform one with multi-edge cells. */
int fcfcg_axis_ftab(fcfcg_axis *a, int allow_log);
/* Build the tile kernel's edge tables of an axis for values up to top;
 * root: of the square roots of the edges (pi of a survey). */
int fcfcg_axis_etab(fcfcg_axis *a, double top, int root);
/* Accessors of the opaque context used by the post-processing code. */
const fcfcg_bins *fcfcg_ctx_bins(const fcfcg_ctx *c);
const double *fcfcg_ctx_box_raw(const fcfcg_ctx *c);

/* ------------------------------------------------------------------------ */
/* Launch parameters of the counting kernels (passed by value).             */

typedef struct {
  /* sorted catalogue on the device */
  const float *l4;       /* float4 per point: local x, y, z, scaled weight */
  const int *wq;         /* int2 per point: round(w 2^30) and the float bits
                            of the remainder, w scaled to |w| <= 1 */
  const double *x, *y, *z, *s, *w;   /* rescaled FP64, |x|^2, weight */
  const uint32_t *id;    /* input index */
  /* blocks of at most 32 points of a cell: two float4 each, (box centre,
   * bits of the first sorted index) and (half extents, bits of the count; 0
   * for a place left unused); bstart: the cells' first blocks (ncell + 1); bcell: (cell, catalogue of
   * a batch) per block */
  const float *blk;
  const uint32_t *bstart, *bcell;
  int wexp;              /* weights scaled by 2^-wexp (for a count graph, which
                            compares its plans, as the sort's scale is captured) */
} fcfcg_dcat;

/* One catalogue of a batch (periodic boxes; all share the bins and the
 * cell stencil, each has its own box, grid and histogram). */
typedef struct {
  int ncell[3];
  uint32_t cell_base;    /* global index of the catalogue's first cell */
  double cw[3];          /* cell widths (rescaled units) */
  double box[3];         /* rescaled box */
  unsigned long long *gcnt;    /* ntot counts */
  unsigned long long *gwt;     /* 2 * ntot: lo, hi words of int128 */
} fcfcg_mock;

typedef struct {
  int geometry, bintype, isauto, withwt;
  int ncell[3];
  double cw[3], lo[3], box[3];
  float cwf[3];
  /* stencil: nsten entries of int4 (ox, oy, oz, 0) and float4 (-o * cw) */
  int nsten;
  const int *sten;
  const float *stenD;
  uint32_t *item_head;
  /* tile kernel: the number of A blocks (device), log2 of the parts a
   * block's tiles are dealt to, slack of the block box distance, and for a
   * batch the catalogues' first cells (their number + 1) */
  const uint32_t *nblk_dev;
  int pshift, tshift;
  uint32_t nsplit;       /* the blocks dealt in parts, the last ones */
  float box_eps;
  const uint32_t *mbase;
  fcfcg_dcat A, B;
  /* bins */
  int ns, nmu, np;
  long ntot;
  float s_lim, p_lim;          /* values at/above: out of range for sure */
  /* survey (s_perp, pi): a pair with |d.u_b| >= los_p + (los_pr + los_h
   * s^2) / |x_b| (u_b = x_b / |x_b|) has pi >= pi_max for sure; the test
   * is skipped for |x_b|^2 <= los_r2min */
  float los_p, los_pr, los_h, los_r2min;
  /* the tile kernel's linear bins: column rn((s + tl_s0) tl_inv), an edge
   * within the window at a distance >= tl_h from the column's middle; mu:
   * rn((mu + tl_q0) nmu) and >= tl_qc - tl_q1 / s; |x_b|^2 below near2: the line of sight is
   * tested per pair.  Shared histogram: hcols columns per row, bin (0, 0) at
   * column hcol0, row hrow0; hrows rows of bins; hlen in all */
  int tlin, tplin;             /* linear s bins; linear pi bins */
  float tl_inv, tl_s0, tl_h, tl_q0, tl_q1, tl_qc, near2;
  /* linear pi bins: row rn((pi + tl_p0) tl_pinv), window at tl_hp (pi by
   * table: its window); tables: the window of s^2 or s_perp^2 is tl_ea s^2 +
   * tl_eb */
  float tl_p0, tl_pinv, tl_hp, tl_ea, tl_eb;
  /* s^2 or s_perp^2, and pi, of an unambiguous pair outside the bins: below
   * tl_slo, tl_plo, or (survey s_perp^2) from tl_shi on */
  float tl_slo, tl_shi, tl_plo;
  /* edge tables (float2 per cell: the edge, 1.5 2^23 + the column below it):
   * cell = FP32 bits >> lg, from off on; in use from the skip-th, the last
   * entry being entry *_last, for all values below */
  const float *se, *pe;
  int nse, npe, se_lg, pe_lg, se_off, pe_off, se_skip, pe_skip, se_last,
      pe_last;
  int hcols, hcol0, hrow0, hrows, hlen;
  int hlog, hwords;            /* in 2^hlog copies: hwords = hlen << hlog */
  float m2min;                 /* survey: |m|^2 below (next to the observer):
                                  mu and pi^2 are rechecked */
  int tzero;                   /* stencil index of the zero offset */
  float fnmu;
  /* FP64 reference binning */
  const uint16_t *rs, *rp;
  long rsoff, rpoff, nrs, nrp;
  const double *s2edge, *pedge;
  double s2min, s2max, pmin, pmax;
  int smin0, pmin0;
  int mu_one;                  /* WITH_MU_ONE: clamp the mu bin, not drop */
  /* outputs */
  unsigned long long *gcnt;    /* ntot counts */
  unsigned long long *gwt;     /* 2 * ntot: lo, hi words of int128 */
  double *gwd;                 /* FP64 sums (FP64 path): fcfcg_gwd_copies of
                                  ntot, the sum of all in the first */
  /* recheck queue: uint4 (a, b, code, 0) */
  uint32_t *queue;
  unsigned long long *qcount;  /* fill: 64 bits, so it cannot wrap */
  uint32_t qcap;
  unsigned long long *stats;   /* [0] candidates (pairs of the fours of A
                                  tested against a block) [1] in-range [2] recheck
                                  [3] inline rechecks [4] blocks */
  int hist_smem;               /* histogram in shared memory */
  /* unweighted shared histogram: pairs a CTA adds between hand-overs to
   * the global counters, at most 2^32 - 1 (u32 bins) */
  unsigned long long hs_limit;
  /* batch of catalogues (NULL: one catalogue pair) */
  const fcfcg_mock *mocks;
  /* adjoint of the weighted counts: gadj[ntot] in, FP64 gradients per
   * sorted point out (dA, dB; the same array for auto counts) */
  int adjoint;
  const double *gadj;
  double *dA, *dB;
  /* the FP32 kernel: per shared bin (hlen, and 32 zeros) the cotangent
   * scaled to at most 1 as round(g 2^30) and the remainder's float bits; a
   * term's unit in the gradients of A and of B */
  const int *gtab;
  double gunitA, gunitB;
} fcfcg_launch;

/* Copies of the FP64 sums the CTAs spread their shared ones over: a bin's
 * chain of additions in memory, of rounding errors each as large as the sum's,
 * is as much shorter.  One where the sums do not fit in shared memory. */
#define FCFCG_GWD_COPIES 32
#define fcfcg_gwd_copies(ntot) ((ntot) <= 25600 ? FCFCG_GWD_COPIES : 1)

/* Launchers implemented in the .cu files; return 0 or a CUDA error code. */
/* Rescale and |x|^2 (surveys); out[0..5] the bounding box (order-preserving
 * keys, min then max), out[6] max |w| bits and, with w, out[7] the sum of the
 * weights (a double, in a fixed order).  out: memory the device can write;
 * acc: 8 words, three ~0 and five 0, left so; partial:
 * fcfcg_prep_partials() doubles of scratch. */
int fcfcg_k_prep(void *stream, size_t n, const double *x, const double *y,
    const double *z, const double *w, double rescale, int survey,
    double *ox, double *oy, double *oz, double *os, double *ow,
    unsigned long long *acc, double *partial, unsigned long long *out);
size_t fcfcg_prep_partials(void);
/* Sub-cell bits of a grid of ncell cells holding npoint points: 6 (4 x 4
 * x 4 sub-cells), 3 (2 x 2 x 2) or 0; the sort then uses (ncell << sb) fine
 * counters.  curve: those of the sort along a Hilbert curve, also 9, 12 and
 * 15 where cells hold many points. */
int fcfcg_grid_sub_bits(size_t ncell, size_t npoint);
int fcfcg_grid_curve_bits(size_t ncell, size_t npoint);
/* Buffers of a sort into a grid of nc cells (sb sub-cell bits) of n points:
 * scratch cell_of, rank (n), key (float4, n), cfill and fstart ((nc << sb) +
 * 1), scan_tmp (fcfcg_scan_tmp_len of that); results cstart and bstart (nc +
 * 1), the sorted arrays (n) and blk, bcell (fcfcg_max_blocks). */
typedef struct {
  uint32_t *cell_of, *rank, *cfill, *fstart, *scan_tmp;
  float *key;
  uint32_t *cstart, *bstart;
  float *l4;
  int *wq;
  double *sx, *sy, *sz, *ss, *sw;
  uint32_t *sid;
  float *blk;
  uint32_t *bcell;
} fcfcg_sort;

/* Sort into the grid: cells in order, within a cell runs along a Hilbert
 * curve of its sub-cells, within a run blocks of 32 (prep.cu:k_runs).
 * cstart[0..nc]: the cells' first sorted points; bstart: their first blocks;
 * blk, bcell: see fcfcg_dcat.  *nl counts the launches (and below). */
size_t fcfcg_max_blocks(size_t n, size_t ncell);
int fcfcg_k_grid(void *stream, size_t n, const double *x, const double *y,
    const double *z, const double *s, const double *w, int has_w, int wexp,
    const int ncell[3], const double cw[3], const double lo[3], int sb,
    const fcfcg_sort *S, uint64_t *nl);
/* One catalogue of a batch for the preparation kernels: its inputs (device
 * or GPU-readable host memory), its place o in the batch slot, its first
 * tile (tiles of fcfcg_batch_tile() points, numbered across the batch) and,
 * once its range checks pass (live), its grid and weight scale. */
typedef struct {
  const double *x, *y, *z, *w;
  size_t o, n;
  uint32_t tile0;
  int live, wexp;
  int ncell[3];
  uint32_t cell_base;
  double cw[3], inv[3];  /* cell widths and their reciprocals */
} fcfcg_prep_cat;

size_t fcfcg_batch_tile(void);
/* Every catalogue rescaled into the slot arrays o*; per catalogue a,
 * bstat[8a + 0..5] its bounding box (order-preserving keys, min then max;
 * initialised by the caller to ~0 and 0), bstat[8a + 6] max |w| bits and,
 * with weights, bstat[8a + 7] the weight sum (a double, in a fixed order;
 * partial: ntile doubles of scratch). */
int fcfcg_k_prep_batch(void *stream, const fcfcg_prep_cat *d_cat, int ncat,
    uint32_t ntile, double rescale, int withwt, double *ox, double *oy,
    double *oz, double *ow, unsigned long long *bstat, double *partial);
/* The same for a batch: every live catalogue's cells numbered from its
 * cell_base (mbase: the catalogues' first cells, ncat + 1), one sorted array;
 * the id of slot point i is i. */
int fcfcg_k_grid_batch(void *stream, const fcfcg_prep_cat *d_cat, int ncat,
    uint32_t ntile, size_t ncell, size_t n, const uint32_t *mbase, int sb,
    const double *x, const double *y, const double *z, const double *w,
    int has_w, const fcfcg_sort *S, uint64_t *nl);
/* out[sid[p]] = in[p] for p < n (sorted order back to input order). */
int fcfcg_k_unsort(void *stream, size_t n, const uint32_t *sid,
    const double *in, double *out);
/* Shared memory of the tile kernel: its tables, and besides them and its
 * histogram (kind: 0 unweighted, 1 weighted, 2 adjoint, 3 all-FP64). */
size_t fcfcg_k_tile32_tab(const fcfcg_launch *L);
size_t fcfcg_k_tile32_stage(int kind);
/* And its histogram's, with a spare word per lane. */
size_t fcfcg_k_tile32_hist(int hwords, int withwt);
/* The count kernel of a launch.  occ: the CTAs per SM of the launches so
 * far (a context's; the last FCFCG_OCC shapes). */
#define FCFCG_OCC 8
typedef struct {
  const void *f[FCFCG_OCC];
  size_t smem[FCFCG_OCC];
  int per_sm[FCFCG_OCC], next;
} fcfcg_occ;
int fcfcg_k_count(void *stream, const fcfcg_launch *L, int precision,
    int nsm, fcfcg_occ *occ, uint64_t *nl);
/* Bits of the coarse cells (dim, cells of 1 / inv_cell from lo) that hold
 * an object, and their number (count). */
int fcfcg_k_occupancy(void *stream, size_t n, const double *x,
    const double *y, const double *z, const double lo[3], const int dim[3],
    const double inv_cell[3], uint32_t *bits, size_t nw,
    unsigned long long *count);
/* FP64 recheck of the queued pairs; the kernels read the queue length on
 * the device, nq_bound (>= it) only sizes the grid. */
int fcfcg_k_recheck(void *stream, const fcfcg_launch *L, uint32_t nq_bound,
    uint64_t *nl);
size_t fcfcg_scan_tmp_len(size_t n);
const char *fcfcg_cuda_errstr(int code);

/* RA/Dec/z conversion (cnvt.c host set-up, cnvt.cu kernels). */
typedef struct {
  double om, ol, ok;     /* Omega_m, Omega_Lambda, Omega_k */
  double widx;           /* 3 (1 + w), 0 for a cosmological constant */
  double c01;            /* SPEED_OF_LIGHT * 0.01 */
  int order;             /* Gauss-Legendre order */
} fcfcg_cnvt_par;
int fcfcg_k_zrange(void *stream, size_t n, const double *z,
    unsigned long long *bits2);
int fcfcg_k_cnvt_integr(void *stream, size_t n, const double *ra,
    const double *dec, const double *z, double *x, double *y, double *zc,
    const fcfcg_cnvt_par *p);
int fcfcg_k_cnvt_spline(void *stream, size_t n, const double *ra,
    const double *dec, const double *z, double *x, double *y, double *zc,
    const double *zs, const double *ds, const double *ypp, size_t nsp,
    unsigned long long *nbad);
/* Converts n objects on `stream` (device pointers, outputs may alias the
 * inputs); *scratch / *scratch_cap is a device buffer the call may grow;
 * *launches counts kernel launches; a message goes to err. */
int fcfcg_cnvt_device(void *stream, size_t n, const double *ra,
    const double *dec, const double *z, double *x, double *y, double *zc,
    const fcfcg_cosmo *cosmo, void **scratch, size_t *scratch_cap,
    int *order, long *launches, char *err, size_t errlen);

#ifdef __cplusplus
}
#endif
#endif

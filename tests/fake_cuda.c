/*
 * fake_cuda.c -- a CUDA runtime and kernel launchers on the host, to compile
 * ctx.c and bins.c against: device memory is host memory whose allocations are
 * tracked, an allocation can be made to fail, and every launch checks that what
 * it is given is allocated, large enough and, where a kernel reads sorted
 * catalogues, sorted since it was allocated.  Used by test_failed_alloc.py.
 */
#include <cuda_runtime_api.h>
#include <math.h>
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include "fcfcg_internal.h"

#define NMAX 65536
static struct { char *p; size_t n; int live, sorted; } blk[NMAX];
static int nblk, fail_at, faults;
static char what[256];

void fake_fail_at(int k) { fail_at = k; }
int fake_faults(void) { return faults; }
void fake_reset(void) { faults = fail_at = 0; }
const char *fake_what(void) { return what; }
int fake_armed(void) { return fail_at > 0; }

static void fault(const char *name) {
  if (!faults++) snprintf(what, sizeof what, "%s", name);
}
static int find(const void *p) {
  for (int i = nblk - 1; i >= 0; i--)
    if (blk[i].live && (const char *) p >= blk[i].p &&
        (const char *) p < blk[i].p + blk[i].n) return i;
  return -1;
}
static int dev(const void *p, size_t n, const char *name) {
  const int i = find(p);
  if (i < 0 || (size_t) ((const char *) p - blk[i].p) + n > blk[i].n) {
    fault(name);
    return -1;
  }
  return i;
}
static void sorted(const void *p, const char *name) {
  const int i = dev(p, 1, name);
  if (i >= 0 && !blk[i].sorted) fault(name);
}

/* (freed memory is kept, so that its address is not handed out again) */
cudaError_t cudaMalloc(void **p, size_t n) {
  if (fail_at && --fail_at == 0) return cudaErrorMemoryAllocation;
  if (nblk == NMAX) abort();
  blk[nblk].p = *p = calloc(1, n < 1 << 26 ? n : 1 << 26);
  blk[nblk].n = n;
  blk[nblk].live = 1;
  blk[nblk++].sorted = 0;
  return cudaSuccess;
}
cudaError_t cudaFree(void *p) {
  if (!p) return cudaSuccess;
  const int i = find(p);
  if (i < 0 || blk[i].p != p) {
    fault("cudaFree");
    return cudaErrorInvalidValue;
  }
  blk[i].live = 0;
  return cudaSuccess;
}
cudaError_t cudaMallocHost(void **p, size_t n) {
  *p = calloc(1, n);
  return cudaSuccess;
}
cudaError_t cudaFreeHost(void *p) {
  free(p);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n,
    enum cudaMemcpyKind k, cudaStream_t st) {
  (void) st;
  if (!n) return cudaSuccess;
  if (k == cudaMemcpyHostToDevice && dev(d, n, "copy to") < 0) return 0;
  if (k == cudaMemcpyDeviceToHost && dev(s, n, "copy from") < 0) return 0;
  memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpy(void *d, const void *s, size_t n,
    enum cudaMemcpyKind k) {
  return cudaMemcpyAsync(d, s, n, k, 0);
}
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t st) {
  (void) st;
  if (n && dev(d, n, "memset") >= 0) memset(d, v, n);
  return cudaSuccess;
}
cudaError_t cudaGetDeviceCount(int *n) { *n = 1; return cudaSuccess; }
cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) { (void) d; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, enum cudaDeviceAttr a, int d) {
  (void) d;
  *v = a == cudaDevAttrMultiProcessorCount ? 152 : 1;
  return cudaSuccess;
}
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t e) { return e ? "error" : "ok"; }
cudaError_t cudaEventCreate(cudaEvent_t *e) { *e = 0; return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t e) { (void) e; return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
  (void) e; (void) s;
  return cudaSuccess;
}
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t a, cudaEvent_t b) {
  (void) a; (void) b;
  *ms = 0;
  return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned f) {
  (void) f;
  *s = 0;
  return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) { (void) s; return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
  (void) s;
  return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t s,
    enum cudaStreamCaptureMode m) {
  (void) s; (void) m;
  return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t s, cudaGraph_t *g) {
  (void) s;
  *g = 0;
  return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *e, cudaGraph_t g,
    unsigned long long f) {
  (void) g; (void) f;
  *e = 0;
  return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t e, cudaStream_t s) {
  (void) e; (void) s;
  return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t g) { (void) g; return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t e) {
  (void) e;
  return cudaSuccess;
}

/* ---- launchers ---- */
const char *fcfcg_cuda_errstr(int e) { return e ? "error" : "ok"; }
size_t fcfcg_prep_partials(void) { return 64; }
size_t fcfcg_batch_tile(void) { return 2048; }
size_t fcfcg_scan_tmp_len(size_t n) { return n / 4096 + 2; }
int fcfcg_grid_curve_bits(size_t nc, size_t n) { (void) nc; (void) n; return 3; }
size_t fcfcg_max_blocks(size_t n, size_t nc) { return n / 32 + nc + 1; }
size_t fcfcg_k_tile32_tab(const fcfcg_launch *L) { (void) L; return 64; }
size_t fcfcg_k_tile32_stage(int kind) { (void) kind; return 32768; }
size_t fcfcg_k_tile32_hist(int hw, int wt) {
  return ((size_t) hw + 32) * (wt ? 8 : 4);
}

static unsigned long long key(double v) {
  unsigned long long b;
  memcpy(&b, &v, 8);
  return b >> 63 ? ~b : b | 0x8000000000000000ull;
}
static void range(const double *x, size_t n, double rescale,
    unsigned long long *lo, unsigned long long *hi) {
  *lo = ~0ull;
  *hi = 0;
  for (size_t i = 0; i < n; i++) {
    const unsigned long long k = key(x[i] * rescale);
    if (k < *lo) *lo = k;
    if (k > *hi) *hi = k;
  }
}
int fcfcg_k_prep(void *st, size_t n, const double *x, const double *y,
    const double *z, const double *w, double rescale, int survey, double *ox,
    double *oy, double *oz, double *os, double *ow, unsigned long long *acc,
    double *partial, unsigned long long *out) {
  const double *in[3] = {x, y, z};
  (void) st; (void) w; (void) survey;
  dev(ox, 8 * n, "prep x"), dev(oy, 8 * n, "prep y"), dev(oz, 8 * n, "prep z");
  dev(os, 8 * n, "prep s"), dev(ow, 8 * n, "prep w");
  dev(acc, 64, "prep acc"), dev(partial, 64, "prep partial");
  for (int k = 0; k < 3; k++) range(in[k], n, rescale, out + k, out + 3 + k);
  const double one = 1;
  memcpy(out + 6, &one, 8);
  memcpy(out + 7, &one, 8);
  return 0;
}
static void grid_check(size_t n, size_t nc, int sb, const fcfcg_sort *S) {
  const size_t nf = nc << sb, mb = fcfcg_max_blocks(n, nc);
  dev(S->cell_of, 4 * n, "cell_of"), dev(S->rank, 4 * n, "rank");
  dev(S->cfill, 4 * nf, "cfill"), dev(S->fstart, 4 * nf + 4, "fstart");
  dev(S->scan_tmp, 4 * fcfcg_scan_tmp_len(nf), "scan_tmp");
  dev(S->key, 16 * n, "key");
  const void *p[] = {S->cstart, S->bstart, S->l4, S->wq, S->sx, S->sy, S->sz,
                     S->sw, S->sid, S->blk, S->bcell, S->ss};
  const size_t m[] = {4 * nc + 4, 4 * nc + 4, 16 * n, 8 * n, 8 * n, 8 * n,
                      8 * n, 8 * n, 4 * n, 32 * mb, 8 * mb, 8 * n};
  for (int k = 0; k < 12; k++) {
    if (!p[k] && k == 11) continue;
    const int i = dev(p[k], m[k], "sorted array");
    if (i >= 0) blk[i].sorted = 1;
  }
}
int fcfcg_k_grid(void *st, size_t n, const double *x, const double *y,
    const double *z, const double *s, const double *w, int has_w, int wexp,
    const int nc[3], const double cw[3], const double lo[3], int sb,
    const fcfcg_sort *S, uint64_t *nl) {
  (void) st; (void) has_w; (void) wexp; (void) cw; (void) lo; (void) nl;
  dev(x, 8 * n, "x"), dev(y, 8 * n, "y"), dev(z, 8 * n, "z");
  if (s) dev(s, 8 * n, "s");
  dev(w, 8 * n, "w");
  grid_check(n, (size_t) nc[0] * nc[1] * nc[2], sb, S);
  return 0;
}
int fcfcg_k_grid_batch(void *st, const fcfcg_prep_cat *cat, int ncat,
    uint32_t ntile, size_t nc, size_t n, const uint32_t *mbase, int sb,
    const double *x, const double *y, const double *z, const double *w,
    int has_w, const fcfcg_sort *S, uint64_t *nl) {
  (void) st; (void) ntile; (void) w; (void) has_w; (void) nl;
  dev(cat, sizeof *cat * ncat, "table"), dev(mbase, 4 * ncat + 4, "mbase");
  dev(x, 8 * n, "x"), dev(y, 8 * n, "y"), dev(z, 8 * n, "z");
  grid_check(n, nc, sb, S);
  return 0;
}
int fcfcg_k_prep_batch(void *st, const fcfcg_prep_cat *cat, int ncat,
    uint32_t ntile, double rescale, int withwt, double *ox, double *oy,
    double *oz, double *ow, unsigned long long *bstat, double *partial) {
  (void) st; (void) withwt; (void) ow;
  dev(cat, sizeof *cat * ncat, "table"), dev(bstat, 64 * ncat, "bstat");
  dev(partial, 8 * ntile, "partial");
  for (int a = 0; a < ncat; a++) {
    const double *in[3] = {cat[a].x, cat[a].y, cat[a].z};
    double *o[3] = {ox, oy, oz};
    for (int k = 0; k < 3; k++) {
      dev(o[k] + cat[a].o, 8 * cat[a].n, "slot");
      range(in[k], cat[a].n, rescale, bstat + 8 * a + k, bstat + 8 * a + 3 + k);
    }
  }
  return 0;
}
int fcfcg_k_count(void *st, const fcfcg_launch *L, int prec, int nsm,
    fcfcg_occ *occ, uint64_t *nl) {
  (void) st; (void) prec; (void) nsm; (void) occ; (void) nl;
  const fcfcg_dcat *D[2] = {&L->A, &L->B};
  for (int k = 0; k < 2; k++) {
    sorted(D[k]->l4, "count l4"), sorted(D[k]->wq, "count wq");
    sorted(D[k]->x, "count x"), sorted(D[k]->w, "count w");
    sorted(D[k]->id, "count id"), sorted(D[k]->blk, "count blk");
    sorted(D[k]->bcell, "count bcell"), sorted(D[k]->bstart, "count bstart");
  }
  dev(L->sten, 16 * (size_t) L->nsten, "stencil");
  dev(L->queue, 16 * (size_t) L->qcap, "queue");
  return 0;
}
int fcfcg_k_recheck(void *st, const fcfcg_launch *L, uint32_t nq,
    uint64_t *nl) {
  (void) st; (void) L; (void) nq; (void) nl;
  return 0;
}
int fcfcg_k_unsort(void *st, size_t n, const uint32_t *sid, const double *in,
    double *out) {
  (void) st;
  sorted(sid, "sid");
  dev(in, 8 * n, "gradient"), dev(out, 8 * n, "gradient");
  return 0;
}
int fcfcg_k_occupancy(void *st, size_t n, const double *x, const double *y,
    const double *z, const double lo[3], const int dim[3],
    const double inv[3], uint32_t *bits, size_t nw,
    unsigned long long *count) {
  (void) st; (void) n; (void) x; (void) y; (void) z; (void) lo; (void) dim;
  (void) inv;
  dev(bits, 4 * nw, "occupancy");
  *count = n;
  return 0;
}
int fcfcg_cnvt_device(void *st, size_t n, const double *ra, const double *dec,
    const double *z, double *x, double *y, double *zc, const fcfcg_cosmo *c,
    void **scratch, size_t *cap, int *order, long *launches, char *err,
    size_t errlen) {
  (void) st; (void) n; (void) ra; (void) dec; (void) z; (void) x; (void) y;
  (void) zc; (void) c; (void) scratch; (void) cap; (void) order;
  (void) launches; (void) err; (void) errlen;
  return 0;
}

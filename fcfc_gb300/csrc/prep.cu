/*
 * prep.cu -- catalogue preparation on the device: rescaling (as FCFC's
 * tree_create does, src/fcfc/2pt_box/build_tree.c:121-131), |x|^2 for
 * surveys (src/fcfc/2pt/build_tree.c:35-133), weight range, bounding box,
 * and the cell grid: a counting sort of the points into cells, stored as
 * SoA FP64 copies plus one float4 per point (FP32 offsets from the cell
 * centre and the scaled high part of the weight) for the FP32 kernels.
 */
#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>

#include "fcfcg_internal.h"

#define PREP_THREADS 256
#define SCAN_THREADS 1024
#define SCAN_ITEMS 4
#define SCAN_TILE (SCAN_THREADS * SCAN_ITEMS)

static int grid_for(size_t n, int threads) {
  size_t b = (n + threads - 1) / threads;
  if (b > 152 * 32) b = 152 * 32;
  if (b < 1) b = 1;
  return (int) b;
}

/* Order-preserving map of a double to an unsigned key.  The bits are taken
 * in PTX: with __double_as_longlong the compiler sets the sign by a negation
 * of the double, which leaves a NaN's alone. */
__device__ __forceinline__ unsigned long long dkey(double v) {
  unsigned long long b;
  asm("mov.b64 %0, %1;" : "=l"(b) : "d"(v));
  return (b >> 63) ? ~b : (b | 0x8000000000000000ull);
}

/* Smallest and largest over the block of lo[k] and hi[k], and the largest of
 * wm, into the accumulators acc[0..2], acc[3..5] and acc[6]: one atomic per
 * block, and only where it would change the value (by then most blocks would
 * not; one per warp, 6 words each, took 73 us for 6e5 points). */
__device__ __forceinline__ void block_range(unsigned long long lo[3],
    unsigned long long hi[3], unsigned long long wm, unsigned long long *acc) {
  __shared__ unsigned long long sh[PREP_THREADS / 32][7];
  const int lane = threadIdx.x & 31;
  for (int o = 16; o > 0; o >>= 1) {
    unsigned long long t;
    for (int k = 0; k < 3; k++) {
      t = __shfl_xor_sync(0xffffffffu, lo[k], o);
      lo[k] = t < lo[k] ? t : lo[k];
      t = __shfl_xor_sync(0xffffffffu, hi[k], o);
      hi[k] = t > hi[k] ? t : hi[k];
    }
    t = __shfl_xor_sync(0xffffffffu, wm, o);
    wm = t > wm ? t : wm;
  }
  if (lane == 0) {
    for (int k = 0; k < 3; k++) {
      sh[threadIdx.x >> 5][k] = lo[k];
      sh[threadIdx.x >> 5][3 + k] = hi[k];
    }
    sh[threadIdx.x >> 5][6] = wm;
  }
  __syncthreads();
  if (threadIdx.x < 7) {
    const int k = threadIdx.x;
    unsigned long long v = sh[0][k];
    for (int i = 1; i < PREP_THREADS / 32; i++) {
      const unsigned long long t = sh[i][k];
      v = k < 3 ? (t < v ? t : v) : (t > v ? t : v);
    }
    const unsigned long long old = *(volatile unsigned long long *) (acc + k);
    if (k < 3) {
      if (v < old) atomicMin(acc + k, v);
    } else if (v > old) {
      atomicMax(acc + k, v);
    }
  }
}

/* The block's sum of v, in a fixed order, by thread 0. */
__device__ __forceinline__ double block_sum(double v) {
  __shared__ double sh[PREP_THREADS];
  sh[threadIdx.x] = v;
  __syncthreads();
  for (int o = PREP_THREADS / 2; o > 0; o >>= 1) {
    if ((int) threadIdx.x < o)
      sh[threadIdx.x] = __dadd_rn(sh[threadIdx.x], sh[threadIdx.x + o]);
    __syncthreads();
  }
  return sh[0];
}

/* A catalogue in one pass: rescaled, |x|^2, its bounding box, max |w| and
 * the sum of the weights, in a fixed order: the blocks' sums, added by the
 * block that finishes last, which also hands the results over and leaves the
 * accumulators as it found them.  (With the box, the sum and the copies as
 * operations of their own, a small catalogue's load was 7 of them.) */
__global__ void k_prep(size_t n, const double *__restrict__ x,
    const double *__restrict__ y, const double *__restrict__ z,
    const double *__restrict__ w, double rescale, int survey,
    double *__restrict__ ox, double *__restrict__ oy, double *__restrict__ oz,
    double *__restrict__ os, double *__restrict__ ow,
    unsigned long long *acc, double *__restrict__ partial,
    unsigned long long *out) {
  __shared__ uint32_t sh_last;
  unsigned long long lo[3] = {~0ull, ~0ull, ~0ull}, hi[3] = {0, 0, 0};
  unsigned long long wm = 0;
  double ws = 0;
  for (size_t i = blockIdx.x * (size_t) blockDim.x + threadIdx.x; i < n;
       i += (size_t) gridDim.x * blockDim.x) {
    double v[3] = {x[i], y[i], z[i]};
    if (rescale != 1)
      for (int k = 0; k < 3; k++) v[k] = __dmul_rn(v[k], rescale);
    ox[i] = v[0];
    oy[i] = v[1];
    oz[i] = v[2];
    if (survey)
      os[i] = __dadd_rn(__dadd_rn(__dmul_rn(v[0], v[0]),
                                  __dmul_rn(v[1], v[1])),
                        __dmul_rn(v[2], v[2]));
    for (int k = 0; k < 3; k++) {
      const unsigned long long q = dkey(v[k]);
      lo[k] = q < lo[k] ? q : lo[k];
      hi[k] = q > hi[k] ? q : hi[k];
    }
    if (w) {
      const double u = w[i];
      ow[i] = u;
      ws = __dadd_rn(ws, u);
      const unsigned long long bits =
          (unsigned long long) __double_as_longlong(fabs(u));
      wm = bits > wm ? bits : wm;
    }
  }
  block_range(lo, hi, wm, acc);
  if (w) {
    const double s = block_sum(ws);
    if (threadIdx.x == 0) partial[blockIdx.x] = s;
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0)
    sh_last = atomicAdd((uint32_t *) (acc + 7), 1u) == gridDim.x - 1u;
  __syncthreads();
  if (!sh_last) return;
  __threadfence();
  double sum = 0;
  if (w) {
    double v = 0;
    for (int i = threadIdx.x; i < (int) gridDim.x; i += PREP_THREADS)
      v = __dadd_rn(v, __ldcg(partial + i));
    __syncthreads();
    sum = block_sum(v);
  }
  if (threadIdx.x < 8) {
    const int k = threadIdx.x;
    out[k] = k < 7 ? __ldcg(acc + k)
                   : (unsigned long long) __double_as_longlong(sum);
    acc[k] = k < 3 ? ~0ull : 0ull;
  }
}

extern "C" size_t fcfcg_prep_partials(void) { return 152 * 32; }

extern "C" int fcfcg_k_prep(void *stream, size_t n, const double *x,
    const double *y, const double *z, const double *w, double rescale,
    int survey, double *ox, double *oy, double *oz, double *os, double *ow,
    unsigned long long *acc, double *partial, unsigned long long *out) {
  if (!n) return 0;
  k_prep<<<grid_for(n, PREP_THREADS), PREP_THREADS, 0,
           (cudaStream_t) stream>>>(n, x, y, z, w, rescale, survey, ox, oy,
                                    oz, os, ow, acc, partial, out);
  return (int) cudaGetLastError();
}

/* ------------------------------------------------------------------------ */
/* Exclusive scan of uint32 (n + 1 outputs: out[n] = total).               */

__device__ __forceinline__ uint32_t block_excl_scan(uint32_t v,
    uint32_t *sh_warp, uint32_t *total) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  uint32_t inc = v;
  for (int o = 1; o < 32; o <<= 1) {
    uint32_t t = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += t;
  }
  if (lane == 31) sh_warp[wid] = inc;
  __syncthreads();
  if (wid == 0) {
    uint32_t s = (lane < (int) (blockDim.x >> 5)) ? sh_warp[lane] : 0;
    uint32_t si = s;
    for (int o = 1; o < 32; o <<= 1) {
      uint32_t t = __shfl_up_sync(0xffffffffu, si, o);
      if (lane >= o) si += t;
    }
    sh_warp[lane] = si - s;
    if (lane == 31) *total = si;
  }
  __syncthreads();
  uint32_t r = sh_warp[wid] + inc - v;
  __syncthreads();
  return r;
}

__global__ void k_scan_tiles(const uint32_t *__restrict__ in, size_t n,
    uint32_t *__restrict__ tile_sum) {
  __shared__ uint32_t shw[32];
  __shared__ uint32_t tot;
  size_t base = (size_t) blockIdx.x * SCAN_TILE;
  uint32_t s = 0;
  for (int k = 0; k < SCAN_ITEMS; k++) {
    size_t i = base + (size_t) k * SCAN_THREADS + threadIdx.x;
    if (i < n) s += in[i];
  }
  block_excl_scan(s, shw, &tot);
  if (threadIdx.x == 0) tile_sum[blockIdx.x] = tot;
}

__global__ void k_scan_sums(uint32_t *__restrict__ tile_sum, size_t ntile) {
  __shared__ uint32_t shw[32];
  __shared__ uint32_t tot;
  uint32_t carry = 0;
  for (size_t b = 0; b < ntile; b += SCAN_THREADS) {
    size_t i = b + threadIdx.x;
    uint32_t v = (i < ntile) ? tile_sum[i] : 0;
    uint32_t e = block_excl_scan(v, shw, &tot);
    if (i < ntile) tile_sum[i] = e + carry;
    carry += tot;
    __syncthreads();
  }
}

__device__ __forceinline__ void scan_put(uint32_t *out, size_t i, uint32_t e,
    int sb, uint32_t *cstart, uint32_t *bstart) {
  out[i] = e;
  if (!cstart || (i & (((size_t) 1 << sb) - 1))) return;
  const size_t c = i >> sb;
  cstart[c] = e;
  if (bstart) bstart[c] = e / 32u + (uint32_t) c;
}

/* The scan itself.  The items before a block: tile_sum[its] where those are
 * scanned (sums 2), else their sum taken here, from the tiles' sums (1) or
 * the items (0).  With cstart, items come (1 << sb) to a cell: cstart[c] the
 * scan at the cells' first items, c = 0..n >> sb, and bstart, if given: the
 * cells' first blocks, numbered with at most one place left unused per cell
 * (floor(cstart / 32) + c grows from cell to cell by more than the cell's
 * points / 32). */
__global__ void k_scan_apply(const uint32_t *__restrict__ in, size_t n,
    const uint32_t *__restrict__ tile_sum, int sums, uint32_t *__restrict__ out,
    int sb, uint32_t *__restrict__ cstart, uint32_t *__restrict__ bstart) {
  __shared__ uint32_t shw[32];
  __shared__ uint32_t tot;
  size_t base = (size_t) blockIdx.x * SCAN_TILE;
  /* each thread owns SCAN_ITEMS consecutive items */
  uint32_t v[SCAN_ITEMS];
  uint32_t s = 0;
  for (int k = 0; k < SCAN_ITEMS; k++) {
    size_t i = base + (size_t) threadIdx.x * SCAN_ITEMS + k;
    v[k] = (i < n) ? in[i] : 0;
    s += v[k];
  }
  uint32_t before = 0;
  if (sums == 2) {
    before = tile_sum[blockIdx.x];
  } else {
    const uint32_t *__restrict__ q = sums ? tile_sum : in;
    const size_t m = sums ? (size_t) blockIdx.x : base;
    uint32_t t = 0;
#pragma unroll 4
    for (size_t i = threadIdx.x; i < m; i += SCAN_THREADS) t += q[i];
    block_excl_scan(t, shw, &tot);
    before = tot;
    __syncthreads();
  }
  uint32_t e = block_excl_scan(s, shw, &tot) + before;
  if (n == 0) scan_put(out, 0, 0, sb, cstart, bstart);
  for (int k = 0; k < SCAN_ITEMS; k++) {
    const size_t i = base + (size_t) threadIdx.x * SCAN_ITEMS + k;
    if (i >= n) break;
    scan_put(out, i, e, sb, cstart, bstart);
    e += v[k];
    if (i == n - 1) scan_put(out, n, e, sb, cstart, bstart);
  }
}

extern "C" size_t fcfcg_scan_tmp_len(size_t n) {
  return (n + SCAN_TILE - 1) / SCAN_TILE + 1;
}

/* out[0..n] = exclusive scan of in[0..n-1], out[n] = total; sb, cstart and
 * bstart as k_scan_apply.  One launch up to 8 tiles, where each block adds
 * up the items before its own; two up to 4096, where each adds up the tiles'
 * sums (16 KB from L2); else three.  *nl counts them. */
static int scan_u32(cudaStream_t s, const uint32_t *in, size_t n,
    uint32_t *out, uint32_t *tmp, uint64_t *nl, int sb = 0,
    uint32_t *cstart = NULL, uint32_t *bstart = NULL) {
  size_t ntile = (n + SCAN_TILE - 1) / SCAN_TILE;
  const int sums = ntile <= 8 ? 0 : (ntile <= 4096 ? 1 : 2);
  if (sums) k_scan_tiles<<<(unsigned) ntile, SCAN_THREADS, 0, s>>>(in, n, tmp);
  if (sums == 2) k_scan_sums<<<1, SCAN_THREADS, 0, s>>>(tmp, ntile);
  k_scan_apply<<<(unsigned) (ntile ? ntile : 1), SCAN_THREADS, 0, s>>>(
      in, n, tmp, sums, out, sb, cstart, bstart);
  *nl += (uint64_t) sums + 1;
  return (int) cudaGetLastError();
}

/* ------------------------------------------------------------------------ */
/* Cell grid.                                                               */

/*
 * The fine index of a point: its global cell (cells of one grid numbered
 * from cell_base), shifted left by sb = 3 r, and its sub-cell (2^r per axis)
 * along a Hilbert curve.  Sorting by the fine index keeps each cell's points
 * contiguous and orders them so that runs of consecutive points (the count
 * kernels' blocks) are compact.  A point's place along an axis is the
 * integer part of (v - lo) 2^r / cw, clamped: with the reciprocal's rounding
 * a point within an ulp of a cell's face may go to either side, which the
 * count kernels' cell margins cover.
 */
struct FineGrid {
  int n[3];
  double inv[3], lo[3];      /* 2^r / cell width */
  uint32_t base;
  int r;
};

static FineGrid fine_grid(const int n[3], const double cw[3],
    const double lo[3], int sb) {
  FineGrid g;
  g.r = sb / 3;
  for (int k = 0; k < 3; k++) {
    g.n[k] = n[k];
    g.inv[k] = (double) (1 << g.r) / cw[k];
    g.lo[k] = lo[k];
  }
  g.base = 0;
  return g;
}

/* Index of a sub-cell along the Hilbert curve of 2^r sub-cells per axis,
 * by J. Skilling's transposition (AIP Conf. Proc. 707, 381, 2004): the axes
 * are rotated and reflected from the highest bit down, Gray-decoded, and
 * their bits interleaved. */
__device__ __forceinline__ uint32_t hilbert3(uint32_t x, uint32_t y,
    uint32_t z, int r) {
  uint32_t X[3] = {x, y, z};
  for (uint32_t Q = 1u << (r - 1); Q > 1; Q >>= 1) {
    const uint32_t P = Q - 1;
#pragma unroll
    for (int i = 0; i < 3; i++) {
      if (X[i] & Q) {
        X[0] ^= P;
      } else {
        const uint32_t t = (X[0] ^ X[i]) & P;
        X[0] ^= t;
        X[i] ^= t;
      }
    }
  }
  X[1] ^= X[0];
  X[2] ^= X[1];
  uint32_t t = 0;
  for (uint32_t Q = 1u << (r - 1); Q > 1; Q >>= 1)
    if (X[2] & Q) t ^= Q - 1;
  uint32_t h = 0;
  for (int b = r - 1; b >= 0; b--)
#pragma unroll
    for (int i = 0; i < 3; i++) h = (h << 1) | (((X[i] ^ t) >> b) & 1u);
  return h;
}

__device__ __forceinline__ uint32_t fine_of_point(const FineGrid &g,
    double a, double b, double d) {
  const double v[3] = {a, b, d};
  int c[3];
  uint32_t s[3];
#pragma unroll
  for (int k = 0; k < 3; k++) {
    int X = __double2int_rd((v[k] - g.lo[k]) * g.inv[k]);
    const int top = (g.n[k] << g.r) - 1;
    X = X < 0 ? 0 : (X > top ? top : X);
    c[k] = X >> g.r;
    s[k] = (uint32_t) X & ((1u << g.r) - 1u);
  }
  const uint32_t cell = g.base +
      ((uint32_t) c[2] * g.n[1] + c[1]) * g.n[0] + c[0];
  return g.r ? (cell << (3 * g.r)) | hilbert3(s[0], s[1], s[2], g.r) : cell;
}

__global__ void k_cell(size_t n, const double *__restrict__ x,
    const double *__restrict__ y, const double *__restrict__ z,
    const FineGrid g, uint32_t *__restrict__ cell_of,
    uint32_t *__restrict__ rank, uint32_t *__restrict__ count) {
  for (size_t i = blockIdx.x * (size_t) blockDim.x + threadIdx.x; i < n;
       i += (size_t) gridDim.x * blockDim.x) {
    const uint32_t c = fine_of_point(g, x[i], y[i], z[i]);
    cell_of[i] = c;
    rank[i] = atomicAdd(count + c, 1u);
  }
}

/* Every point to its place by cell and sub-cell: FP32 coordinates (for the
 * ordering within a run, k_runs) and the input index. */
__global__ void k_keys(size_t n, const double *__restrict__ x,
    const double *__restrict__ y, const double *__restrict__ z,
    const uint32_t *__restrict__ cell_of, const uint32_t *__restrict__ rank,
    const uint32_t *__restrict__ fstart, float4 *__restrict__ key) {
  for (size_t i = blockIdx.x * (size_t) blockDim.x + threadIdx.x; i < n;
       i += (size_t) gridDim.x * blockDim.x)
    key[fstart[cell_of[i]] + rank[i]] = make_float4((float) x[i], (float) y[i],
        (float) z[i], __uint_as_float((uint32_t) i));
}

__global__ void k_block_count(const uint32_t *__restrict__ cstart,
    uint32_t ncell, uint32_t *__restrict__ count) {
  for (uint32_t c = blockIdx.x * blockDim.x + threadIdx.x; c < ncell;
       c += gridDim.x * blockDim.x)
    count[c] = (cstart[c + 1] - cstart[c] + 31u) / 32u;
}

/*
 * The sorted arrays and the blocks.  A cell's points come in runs of at most
 * RUN_LEN along the Hilbert curve; a team of W warps orders a run so that
 * each block of 32 has a compact box: it is halved along its longest axis,
 * the halves along theirs, down to 32 (a bitonic sort of 23-bit coordinates
 * and 9-bit indices in registers, 16 / W per lane).  Consecutive runs of 32
 * points of the curve itself have boxes of about twice the volume; with this
 * order the tiles of a uniform box fell by a fifth.  Then the run is gathered
 * from the input arrays and written in order: the FP32 offsets from the cell
 * centre and the weight's scaled high part (l4), the weight's fixed-point
 * split (wq), FP64 copies and ids, and the blocks' boxes of the FP32 offsets
 * (half extents rounded up).
 *
 * Bound by latency unless there are many runs: one warp per run took 30 us
 * for any number of points up to 1e5 (16 gathers one after the other, 40
 * steps of the sort on 16 keys a lane); four warps share both: 15 us for
 * 2e3 points, 22 us for 1e5 (31 before), 45 for 6e5 (65).  One warp where
 * cells hold few points.
 *
 * Teams: groups of `group` consecutive cells, `share` teams to a group, which
 * deal the cells' runs among themselves.
 */
#define RUN_LEN 512
#define RUN_WARPS 4
struct RunArgs {
  const uint32_t *cstart, *bstart;
  uint32_t ncell;
  uint32_t group, share;
  const float4 *key;
  const double *x, *y, *z, *s, *w;
  int has_w, wexp;
  int nx, ny;
  double cw[3], lo[3];
  const fcfcg_prep_cat *cat;      /* a batch: per catalogue */
  const uint32_t *mbase;
  int ncat;
  float4 *l4;
  int2 *wq;
  double *sx, *sy, *sz, *ss, *sw;
  uint32_t *sid;
  float4 *blk;
  uint2 *bcell;
};
struct RunSh {
  float c[3][RUN_LEN];
  uint32_t id[RUN_LEN];
  uint16_t ord[RUN_LEN];
};
/* a team of four: keys to exchange, and the warps' ranges */
struct RunX {
  uint32_t k[2][RUN_LEN];
  float r[RUN_WARPS][6];
};

template <int W>
__device__ __forceinline__ void team_sync() {
  if (W == 1) __syncwarp();
  else __syncthreads();
}

/* Compare-exchange of keys i and i ^ J of a lane, ascending. */
template <int J, int E>
__device__ __forceinline__ void run_step(uint32_t k[E]) {
#pragma unroll
  for (int i = 0; i < E; i++)
    if (!(i & J)) {
      const uint32_t a = k[i], b = k[i | J];
      k[i] = a < b ? a : b;
      k[i | J] = a < b ? b : a;
    }
}
template <int E>
__device__ __forceinline__ void run_steps(uint32_t k[E]) {
  if (E > 8) run_step<8, E>(k);
  if (E > 4) run_step<4, E>(k);
  run_step<2, E>(k);
  run_step<1, E>(k);
}

/* Sort segments of S keys (thread t's are E t to E t + E - 1), ascending;
 * S = E .. 512. */
template <int W>
__device__ __forceinline__ void run_sort(uint32_t k[16 / W], int S, int t,
    RunX *X) {
  constexpr int E = 16 / W;
  /* bitonic runs within the thread: descending where bit K of the index is
   * set (the keys complemented) */
#pragma unroll
  for (int K = 2; K < E; K <<= 1) {
#pragma unroll
    for (int i = 0; i < E; i++)
      if (i & K) k[i] = ~k[i];
    if (K > 4) run_step<4, E>(k);
    if (K > 2) run_step<2, E>(k);
    run_step<1, E>(k);
#pragma unroll
    for (int i = 0; i < E; i++)
      if (i & K) k[i] = ~k[i];
  }
  int buf = 0;
#pragma unroll 1
  for (int K = E; K <= S; K <<= 1) {
    const uint32_t m = (K < S && ((t * E) & K)) ? 0xffffffffu : 0u;
#pragma unroll
    for (int i = 0; i < E; i++) k[i] ^= m;
#pragma unroll 1
    for (int o = K / (2 * E); o > 0; o >>= 1) {
      const bool low = !(t & o);
      if (W > 1 && o >= 32) {
        /* across warps */
        uint32_t *x = X->k[buf];
        buf ^= 1;
        *(uint4 *) (x + E * t) = make_uint4(k[0], k[1], k[2], k[3]);
        __syncthreads();
        const uint4 q = *(const uint4 *) (x + E * (t ^ o));
        const uint32_t b[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
        for (int i = 0; i < 4; i++)
          k[i] = (low == (k[i] < b[i])) ? k[i] : b[i];
      } else {
#pragma unroll
        for (int i = 0; i < E; i++) {
          const uint32_t b = __shfl_xor_sync(0xffffffffu, k[i], o);
          k[i] = (low == (k[i] < b)) ? k[i] : b;
        }
      }
    }
    run_steps<E>(k);
#pragma unroll
    for (int i = 0; i < E; i++) k[i] ^= m;
  }
}

/* The order of one run, the n points from key[a] on. */
template <int W>
__device__ __forceinline__ void run_order(RunSh *S, RunX *X, const float4 *key,
    uint32_t a, int n, int t) {
  constexpr int E = 16 / W, LMIN = W == 1 ? 16 : 8;
  team_sync<W>();
  for (int i = t; i < n; i += 32 * W) {
    const float4 v = key[a + i];
    S->c[0][i] = v.x;
    S->c[1][i] = v.y;
    S->c[2][i] = v.z;
    S->id[i] = __float_as_uint(v.w);
    S->ord[i] = (uint16_t) i;
  }
  team_sync<W>();
  if (n <= 4) return;
  uint32_t k[E];
#pragma unroll
  for (int i = 0; i < E; i++) k[i] = (uint32_t) (E * t + i);
#pragma unroll 1
  for (int L = RUN_LEN; L >= LMIN; L >>= 1) {
    if (n <= L / 2) continue;       /* all in the first half already */
    /* the longest axis of each segment of L */
    float lo[3] = {3e38f, 3e38f, 3e38f}, hi[3] = {-3e38f, -3e38f, -3e38f};
#pragma unroll
    for (int i = 0; i < E; i++) {
      const int e = (int) (k[i] & (RUN_LEN - 1u));
      if (e < n)
#pragma unroll
        for (int d = 0; d < 3; d++) {
          const float v = S->c[d][e];
          lo[d] = fminf(lo[d], v);
          hi[d] = fmaxf(hi[d], v);
        }
    }
    for (int o = L / (2 * E) < 16 ? L / (2 * E) : 16; o > 0; o >>= 1)
#pragma unroll
      for (int d = 0; d < 3; d++) {
        lo[d] = fminf(lo[d], __shfl_xor_sync(0xffffffffu, lo[d], o));
        hi[d] = fmaxf(hi[d], __shfl_xor_sync(0xffffffffu, hi[d], o));
      }
    if (W > 1 && L > 32 * E) {
      const int w = t >> 5, nw = L / (32 * E);
      __syncthreads();
      if ((t & 31) == 0)
#pragma unroll
        for (int d = 0; d < 3; d++) {
          X->r[w][d] = lo[d];
          X->r[w][3 + d] = hi[d];
        }
      __syncthreads();
      for (int q = w & ~(nw - 1), e = q + nw; q < e; q++)
#pragma unroll
        for (int d = 0; d < 3; d++) {
          lo[d] = fminf(lo[d], X->r[q][d]);
          hi[d] = fmaxf(hi[d], X->r[q][3 + d]);
        }
    }
    const float ex = hi[0] - lo[0], ey = hi[1] - lo[1], ez = hi[2] - lo[2];
    const int d = (ex >= ey && ex >= ez) ? 0 : (ey >= ez ? 1 : 2);
    const float l = lo[d], w = hi[d] - lo[d];
    const float f = w > 0 ? 8388606.f / w : 0.f;
#pragma unroll
    for (int i = 0; i < E; i++) {
      const uint32_t e = k[i] & (RUN_LEN - 1u);
      uint32_t q = 0x7fffffu;
      if ((int) e < n) {
        q = (uint32_t) ((S->c[d][e] - l) * f);
        q = q < 0x7ffffeu ? q : 0x7ffffeu;
      }
      k[i] = q << 9 | e;
    }
    run_sort<W>(k, L, t, X);
  }
#pragma unroll
  for (int i = 0; i < E; i++)
    S->ord[E * t + i] = (uint16_t) (k[i] & (RUN_LEN - 1u));
  team_sync<W>();
}

template <int BATCH, int W>
__global__ void __launch_bounds__(32 * RUN_WARPS) k_runs(const RunArgs A) {
  static_assert(W == 1 || W == RUN_WARPS, "a team is a warp or the block");
  __shared__ RunSh sh[RUN_WARPS / W];
  __shared__ __align__(16) unsigned char shx[W > 1 ? sizeof(RunX) : 16];
  RunX *X = (RunX *) shx;
  const int lane = threadIdx.x & 31, wt = W > 1 ? threadIdx.x >> 5 : 0;
  const int t = W > 1 ? (int) threadIdx.x : lane;
  RunSh *S = sh + (W > 1 ? 0 : threadIdx.x >> 5);
  const uint32_t wid = W > 1 ? blockIdx.x
      : blockIdx.x * RUN_WARPS + (threadIdx.x >> 5);
  const uint32_t r0 = wid % A.share, c0 = wid / A.share * A.group;
  if (c0 >= A.ncell) return;
  const uint32_t c1 = c0 + A.group < A.ncell ? c0 + A.group : A.ncell;
  for (uint32_t c = c0; c < c1; c++) {
    const uint32_t a = __ldg(A.cstart + c), n = __ldg(A.cstart + c + 1) - a;
    const uint32_t b = __ldg(A.bstart + c), nb = (n + 31u) / 32u;
    const uint32_t nrun = (n + RUN_LEN - 1u) / RUN_LEN;
    const bool gap = r0 == 0 && __ldg(A.bstart + c + 1) - b > nb;
    if (r0 >= nrun && !gap) continue;
    int nx = A.nx, ny = A.ny, wexp = A.wexp;
    uint32_t lc = c, mk = 0;
    double cw[3] = {A.cw[0], A.cw[1], A.cw[2]},
           lo[3] = {A.lo[0], A.lo[1], A.lo[2]};
    if (BATCH) {
      int l = 0, h = A.ncat;        /* last l with mbase[l] <= c */
      while (h - l > 1) {
        const int mid = (l + h) >> 1;
        if (__ldg(A.mbase + mid) <= c) l = mid;
        else h = mid;
      }
      mk = (uint32_t) l;
      const fcfcg_prep_cat *C = A.cat + l;
      nx = C->ncell[0];
      ny = C->ncell[1];
      wexp = C->wexp;
      lc = c - C->cell_base;
      for (int k = 0; k < 3; k++) {
        cw[k] = C->cw[k];
        lo[k] = 0.0;
      }
    }
    if (gap && t == 0) {
      /* the place left unused: far from everything, no points */
      A.blk[2 * (size_t) (b + nb)] = make_float4(1e30f, 1e30f, 1e30f, 0.f);
      A.blk[2 * (size_t) (b + nb) + 1] = make_float4(0.f, 0.f, 0.f, 0.f);
      A.bcell[b + nb] = make_uint2(c, mk);
    }
    const double cc[3] = {
        lo[0] + ((double) (int) (lc % (uint32_t) nx) + 0.5) * cw[0],
        lo[1] + ((double) (int) ((lc / (uint32_t) nx) % (uint32_t) ny) + 0.5) * cw[1],
        lo[2] + ((double) (int) (lc / ((uint32_t) nx * (uint32_t) ny)) + 0.5) * cw[2]};
    for (uint32_t r = r0; r < nrun; r += A.share) {
      const uint32_t q0 = r * RUN_LEN;
      const int m = (int) (n - q0 < RUN_LEN ? n - q0 : RUN_LEN);
      run_order<W>(S, X, A.key, a + q0, m, t);
      /* blocks j = wt, wt + W, ..., up to four gathers in flight */
#pragma unroll 1
      for (int jb = 32 * wt; jb < m; jb += 128 * W) {
        double v[4][3], wv[4], sv[4];
        uint32_t id[4];
#pragma unroll
        for (int u = 0; u < 4; u++) {
          const int j = jb + 32 * W * u + lane;
          wv[u] = 1.0;
          if (j < m) {
            const uint32_t i = id[u] = S->id[S->ord[j]];
            v[u][0] = __ldg(A.x + i);
            v[u][1] = __ldg(A.y + i);
            v[u][2] = __ldg(A.z + i);
            if (A.has_w) wv[u] = __ldg(A.w + i);
            if (A.ss) sv[u] = __ldg(A.s + i);
          }
        }
#pragma unroll
        for (int u = 0; u < 4; u++) {
          const int j0 = jb + 32 * W * u, j = j0 + lane;
          if (j0 >= m) break;
          float mn[3] = {3e38f, 3e38f, 3e38f}, mx[3] = {-3e38f, -3e38f, -3e38f};
          const uint32_t pos = a + q0 + (uint32_t) j;
          if (j < m) {
            double ws = wv[u];
            int wi = 1 << 30;
            float wr = 0.f;
            if (A.has_w) {
              ws = ldexp(wv[u], -wexp);          /* |ws| <= 1 */
              wi = (int) __double2ll_rn(ws * 1073741824.0);
              wr = (float) (ws - (double) wi * (1.0 / 1073741824.0));
            }
            float4 p;
            p.x = (float) (v[u][0] - cc[0]);
            p.y = (float) (v[u][1] - cc[1]);
            p.z = (float) (v[u][2] - cc[2]);
            p.w = (float) ws;
            A.l4[pos] = p;
            A.wq[pos] = make_int2(wi, __float_as_int(wr));
            A.sx[pos] = v[u][0];
            A.sy[pos] = v[u][1];
            A.sz[pos] = v[u][2];
            if (A.ss) A.ss[pos] = sv[u];
            A.sw[pos] = wv[u];
            A.sid[pos] = id[u];
            mn[0] = mx[0] = p.x;
            mn[1] = mx[1] = p.y;
            mn[2] = mx[2] = p.z;
          }
#pragma unroll
          for (int o = 16; o > 0; o >>= 1)
#pragma unroll
            for (int k = 0; k < 3; k++) {
              mn[k] = fminf(mn[k], __shfl_xor_sync(0xffffffffu, mn[k], o));
              mx[k] = fmaxf(mx[k], __shfl_xor_sync(0xffffffffu, mx[k], o));
            }
          if (lane == 0) {
            float ce[3], e[3];
            for (int k = 0; k < 3; k++) {
              ce[k] = 0.5f * mn[k] + 0.5f * mx[k];
              e[k] = __fmul_ru(fmaxf(__fsub_ru(mx[k], ce[k]),
                                     __fsub_ru(ce[k], mn[k])), 1.000001f);
            }
            const size_t B = b + (q0 + (uint32_t) j0) / 32u;
            const int cnt = m - j0 < 32 ? m - j0 : 32;
            A.blk[2 * B] = make_float4(ce[0], ce[1], ce[2],
                                       __uint_as_float(pos));
            A.blk[2 * B + 1] = make_float4(e[0], e[1], e[2],
                                           __uint_as_float((uint32_t) cnt));
            A.bcell[B] = make_uint2(c, mk);
          }
        }
      }
      team_sync<W>();
    }
  }
}

/* Teams of k_runs for ncell cells of n points: four warps where cells hold
 * RUN_TEAM points on average; 32 cells to a group where there are many, and
 * twice as many teams to a group as a cell has runs on average. */
#define RUN_TEAM 96
static void launch_runs(RunArgs *A, size_t n, cudaStream_t st) {
  A->group = A->ncell > 32u * 4864u ? 32u : (A->ncell > 4u * 4864u ? 4u : 1u);
  const size_t per = n / A->ncell / RUN_LEN + 1;
  A->share = (uint32_t) (per * 2 < 256 ? per * 2 : 256);
  const uint64_t teams =
      ((uint64_t) A->ncell + A->group - 1) / A->group * A->share;
  if (n >= (size_t) RUN_TEAM * A->ncell) {
    const unsigned nb = (unsigned) teams;
    if (A->cat) k_runs<1, RUN_WARPS><<<nb, 32 * RUN_WARPS, 0, st>>>(*A);
    else k_runs<0, RUN_WARPS><<<nb, 32 * RUN_WARPS, 0, st>>>(*A);
  } else {
    const unsigned nb = (unsigned) ((teams + RUN_WARPS - 1) / RUN_WARPS);
    if (A->cat) k_runs<1, 1><<<nb, 32 * RUN_WARPS, 0, st>>>(*A);
    else k_runs<0, 1><<<nb, 32 * RUN_WARPS, 0, st>>>(*A);
  }
}

extern "C" int fcfcg_grid_sub_bits(size_t ncell, size_t npoint) {
  /* sub-cells where cells hold many points on average, with the fine
   * counters at most ~4 per point (and 32-bit fine indices) */
  const size_t lim = npoint * 4 > ((size_t) 1 << 22) ? npoint * 4
                                                   : ((size_t) 1 << 22);
  if (ncell << 6 <= lim && (ncell << 6) < 0xFFFFFFF0u) return 6;
  if (ncell << 3 <= lim && (ncell << 3) < 0xFFFFFFF0u) return 3;
  return 0;
}

extern "C" int fcfcg_grid_curve_bits(size_t ncell, size_t npoint) {
  /* in coarse cells the finest of 32, 16 or 8 sub-cells per axis with at
   * most 2 fine counters per point, so that clearing and scanning them stays
   * below the cost of moving the points (a sub-cell then holds a few points,
   * well below a block of 32); else 4, 2 or none */
  for (int sb = 15; sb > 6; sb -= 3)
    if (ncell << sb <= npoint * 2 && (ncell << sb) < 0xFFFFFFF0u) return sb;
  return fcfcg_grid_sub_bits(ncell, npoint);
}

/* The blocks' numbering from the cells' points: with gaps (k_scan_apply) unless
 * cells far outnumber the blocks, where it is compacted by a scan. */
static int gaps_ok(size_t n, size_t nc) { return nc <= 4096 || nc <= n / 16; }

extern "C" size_t fcfcg_max_blocks(size_t n, size_t ncell) {
  return n / 32 + (n < ncell && !gaps_ok(n, ncell) ? n : ncell) + 1;
}

/* Fine counts (in cfill) to cell starts, keys and the block numbering. */
static int sort_rest(cudaStream_t st, size_t nc, size_t n, int sb,
    uint32_t *cfill, uint32_t *fstart, uint32_t *scan_tmp, uint32_t *cstart,
    uint32_t *bstart, uint64_t *nl) {
  const int gaps = gaps_ok(n, nc);
  int r = scan_u32(st, cfill, nc << sb, fstart, scan_tmp, nl, sb, cstart,
                   gaps ? bstart : NULL);
  if (r || gaps) return r;
  cudaError_t e;
  k_block_count<<<grid_for(nc, PREP_THREADS), PREP_THREADS, 0, st>>>(
      cstart, (uint32_t) nc, cfill);
  if ((e = cudaGetLastError())) return (int) e;
  ++*nl;
  return scan_u32(st, cfill, nc, bstart, scan_tmp, nl);
}

extern "C" int fcfcg_k_grid(void *stream, size_t n, const double *x,
    const double *y, const double *z, const double *s, const double *w,
    int has_w, int wexp, const int ncell[3], const double cw[3],
    const double lo[3], int sb, const fcfcg_sort *S, uint64_t *nl) {
  cudaStream_t st = (cudaStream_t) stream;
  const size_t nc = (size_t) ncell[0] * ncell[1] * ncell[2];
  cudaError_t e = cudaMemsetAsync(S->cfill, 0, sizeof(uint32_t) * (nc << sb), st);
  if (e) return (int) e;
  if (n) {
    k_cell<<<grid_for(n, PREP_THREADS), PREP_THREADS, 0, st>>>(
        n, x, y, z, fine_grid(ncell, cw, lo, sb), S->cell_of, S->rank, S->cfill);
    if ((e = cudaGetLastError())) return (int) e;
    ++*nl;
  }
  int r = sort_rest(st, nc, n, sb, S->cfill, S->fstart, S->scan_tmp, S->cstart,
                    S->bstart, nl);
  if (r) return r;
  if (n) {
    k_keys<<<grid_for(n, PREP_THREADS), PREP_THREADS, 0, st>>>(
        n, x, y, z, S->cell_of, S->rank, S->fstart, (float4 *) S->key);
    if ((e = cudaGetLastError())) return (int) e;
    ++*nl;
  }
  RunArgs A;
  memset(&A, 0, sizeof A);
  A.cstart = S->cstart;
  A.bstart = S->bstart;
  A.ncell = (uint32_t) nc;
  A.key = (const float4 *) S->key;
  A.x = x;
  A.y = y;
  A.z = z;
  A.s = s;
  A.w = w;
  A.has_w = has_w;
  A.wexp = wexp;
  A.nx = ncell[0];
  A.ny = ncell[1];
  for (int k = 0; k < 3; k++) {
    A.cw[k] = cw[k];
    A.lo[k] = lo[k];
  }
  A.l4 = (float4 *) S->l4;
  A.wq = (int2 *) S->wq;
  A.sx = S->sx;
  A.sy = S->sy;
  A.sz = S->sz;
  A.ss = s ? S->ss : NULL;
  A.sw = S->sw;
  A.sid = S->sid;
  A.blk = (float4 *) S->blk;
  A.bcell = (uint2 *) S->bcell;
  launch_runs(&A, n, st);
  ++*nl;
  return (int) cudaGetLastError();
}

/* ------------------------------------------------------------------------ */
/* Batches: one launch per stage over every catalogue.  Block t handles tile
 * t (BATCH_TILE points of one catalogue); the catalogue table lists each
 * catalogue's first tile, so a block finds its catalogue by bisection. */

#define BATCH_ITEMS 8
#define BATCH_TILE (PREP_THREADS * BATCH_ITEMS)

extern "C" size_t fcfcg_batch_tile(void) { return BATCH_TILE; }

__device__ __forceinline__ int batch_cat(const fcfcg_prep_cat *__restrict__ cat,
    int ncat, uint32_t t) {
  int lo = 0, hi = ncat;          /* the last lo with cat[lo].tile0 <= t */
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (cat[mid].tile0 <= t) lo = mid;
    else hi = mid;
  }
  return lo;
}

/* Rescale every catalogue into the batch slot (as k_prep), with each
 * catalogue's bounding box (order-preserving keys, bstat[8a + 0..5]), max
 * |w| bits (bstat[8a + 6]) and this tile's weight sum in a fixed order
 * (partial[t]). */
__global__ void __launch_bounds__(PREP_THREADS) k_prep_batch(
    const fcfcg_prep_cat *__restrict__ cat, int ncat, double rescale,
    int withwt, double *ox, double *oy, double *oz, double *ow,
    unsigned long long *bstat, double *__restrict__ partial) {
  const uint32_t t = blockIdx.x;
  const int a = batch_cat(cat, ncat, t);
  const fcfcg_prep_cat *C = cat + a;
  const double *x = C->x, *y = C->y, *z = C->z, *w = withwt ? C->w : NULL;
  const size_t o = C->o, n = C->n;
  const size_t i0 = (size_t) (t - C->tile0) * BATCH_TILE;
  const size_t i1 = (i0 + BATCH_TILE < n) ? i0 + BATCH_TILE : n;
  unsigned long long lo[3] = {~0ull, ~0ull, ~0ull}, hi[3] = {0, 0, 0};
  unsigned long long wm = 0;
  double ws = 0;
  for (size_t i = i0 + threadIdx.x; i < i1; i += PREP_THREADS) {
    double v[3] = {x[i], y[i], z[i]};
    if (rescale != 1)
      for (int k = 0; k < 3; k++) v[k] = __dmul_rn(v[k], rescale);
    ox[o + i] = v[0];
    oy[o + i] = v[1];
    oz[o + i] = v[2];
    for (int k = 0; k < 3; k++) {
      const unsigned long long q = dkey(v[k]);
      lo[k] = q < lo[k] ? q : lo[k];
      hi[k] = q > hi[k] ? q : hi[k];
    }
    if (w) {
      const double u = w[i];
      ow[o + i] = u;
      ws = __dadd_rn(ws, u);
      const unsigned long long bits =
          (unsigned long long) __double_as_longlong(fabs(u));
      wm = bits > wm ? bits : wm;
    }
  }
  block_range(lo, hi, wm, bstat + 8 * (size_t) a);
  if (!withwt) return;
  const double s = block_sum(ws);
  if (threadIdx.x == 0) partial[t] = s;
}

/* Block a: catalogue a's weight sum from its tiles' sums, in a fixed order,
 * into bstat[8a + 7] (as a double). */
__global__ void __launch_bounds__(PREP_THREADS) k_sum_batch(
    const fcfcg_prep_cat *__restrict__ cat, int ncat, uint32_t ntile,
    const double *__restrict__ partial, unsigned long long *bstat) {
  const int a = blockIdx.x;
  const uint32_t t0 = cat[a].tile0;
  const uint32_t t1 = (a + 1 < ncat) ? cat[a + 1].tile0 : ntile;
  double v = 0;
  for (uint32_t t = t0 + threadIdx.x; t < t1; t += PREP_THREADS)
    v = __dadd_rn(v, partial[t]);
  const double s = block_sum(v);
  if (threadIdx.x == 0)
    bstat[8 * (size_t) a + 7] =
        (unsigned long long) __double_as_longlong(s);
}

extern "C" int fcfcg_k_prep_batch(void *stream, const fcfcg_prep_cat *d_cat,
    int ncat, uint32_t ntile, double rescale, int withwt, double *ox,
    double *oy, double *oz, double *ow, unsigned long long *bstat,
    double *partial) {
  if (!ncat || !ntile) return 0;
  cudaStream_t st = (cudaStream_t) stream;
  k_prep_batch<<<ntile, PREP_THREADS, 0, st>>>(d_cat, ncat, rescale, withwt,
                                               ox, oy, oz, ow, bstat,
                                               partial);
  cudaError_t e = cudaGetLastError();
  if (e || !withwt) return (int) e;
  k_sum_batch<<<ncat, PREP_THREADS, 0, st>>>(d_cat, ncat, ntile, partial,
                                             bstat);
  return (int) cudaGetLastError();
}

/* Cells of every live catalogue's points (slot arrays x, y, z), numbered
 * from the catalogue's cell_base into the shared count array. */
__global__ void __launch_bounds__(PREP_THREADS) k_cell_batch(
    const fcfcg_prep_cat *__restrict__ cat, int ncat, int sb,
    const double *__restrict__ x, const double *__restrict__ y,
    const double *__restrict__ z, uint32_t *__restrict__ cell_of,
    uint32_t *__restrict__ rank, uint32_t *__restrict__ count) {
  const uint32_t t = blockIdx.x;
  const fcfcg_prep_cat *C = cat + batch_cat(cat, ncat, t);
  if (!C->live) return;
  const size_t o = C->o, n = C->n;
  const size_t i0 = (size_t) (t - C->tile0) * BATCH_TILE;
  const size_t i1 = (i0 + BATCH_TILE < n) ? i0 + BATCH_TILE : n;
  FineGrid g;
  for (int k = 0; k < 3; k++) {
    g.n[k] = C->ncell[k];
    g.inv[k] = C->inv[k] * (double) (1 << (sb / 3));
    g.lo[k] = 0.0;
  }
  g.base = C->cell_base;
  g.r = sb / 3;
  for (size_t i = o + i0 + threadIdx.x; i < o + i1; i += PREP_THREADS) {
    const uint32_t c = fine_of_point(g, x[i], y[i], z[i]);
    cell_of[i] = c;
    rank[i] = atomicAdd(count + c, 1u);
  }
}

/* k_keys for every live catalogue; the index of point i of the slot is i. */
__global__ void __launch_bounds__(PREP_THREADS) k_keys_batch(
    const fcfcg_prep_cat *__restrict__ cat, int ncat,
    const double *__restrict__ x, const double *__restrict__ y,
    const double *__restrict__ z, const uint32_t *__restrict__ cell_of,
    const uint32_t *__restrict__ rank, const uint32_t *__restrict__ fstart,
    float4 *__restrict__ key) {
  const uint32_t t = blockIdx.x;
  const fcfcg_prep_cat *C = cat + batch_cat(cat, ncat, t);
  if (!C->live) return;
  const size_t o = C->o, n = C->n;
  const size_t i0 = (size_t) (t - C->tile0) * BATCH_TILE;
  const size_t i1 = (i0 + BATCH_TILE < n) ? i0 + BATCH_TILE : n;
  for (size_t i = o + i0 + threadIdx.x; i < o + i1; i += PREP_THREADS)
    key[fstart[cell_of[i]] + rank[i]] = make_float4((float) x[i], (float) y[i],
        (float) z[i], __uint_as_float((uint32_t) i));
}

extern "C" int fcfcg_k_grid_batch(void *stream, const fcfcg_prep_cat *d_cat,
    int ncat, uint32_t ntile, size_t ncell, size_t n, const uint32_t *mbase,
    int sb, const double *x, const double *y, const double *z,
    const double *w, int has_w, const fcfcg_sort *S, uint64_t *nl) {
  if (!ncat || !ntile) return 0;
  cudaStream_t st = (cudaStream_t) stream;
  cudaError_t e = cudaMemsetAsync(S->cfill, 0,
                                  sizeof(uint32_t) * (ncell << sb), st);
  if (e) return (int) e;
  k_cell_batch<<<ntile, PREP_THREADS, 0, st>>>(d_cat, ncat, sb, x, y, z,
                                               S->cell_of, S->rank, S->cfill);
  if ((e = cudaGetLastError())) return (int) e;
  ++*nl;
  int r = sort_rest(st, ncell, n, sb, S->cfill, S->fstart, S->scan_tmp,
                    S->cstart, S->bstart, nl);
  if (r) return r;
  k_keys_batch<<<ntile, PREP_THREADS, 0, st>>>(d_cat, ncat, x, y, z,
      S->cell_of, S->rank, S->fstart, (float4 *) S->key);
  if ((e = cudaGetLastError())) return (int) e;
  ++*nl;
  RunArgs A;
  memset(&A, 0, sizeof A);
  A.cstart = S->cstart;
  A.bstart = S->bstart;
  A.ncell = (uint32_t) ncell;
  A.key = (const float4 *) S->key;
  A.x = x;
  A.y = y;
  A.z = z;
  A.w = w;
  A.has_w = has_w;
  A.cat = d_cat;
  A.mbase = mbase;
  A.ncat = ncat;
  A.l4 = (float4 *) S->l4;
  A.wq = (int2 *) S->wq;
  A.sx = S->sx;
  A.sy = S->sy;
  A.sz = S->sz;
  A.sw = S->sw;
  A.sid = S->sid;
  A.blk = (float4 *) S->blk;
  A.bcell = (uint2 *) S->bcell;
  launch_runs(&A, n, st);
  ++*nl;
  return (int) cudaGetLastError();
}

/* Occupancy of a coarse grid over a catalogue's bounding box: one bit per
 * cell that holds an object (the occupied-volume estimate of a survey). */
__global__ void k_occupy(size_t n, const double *__restrict__ x,
    const double *__restrict__ y, const double *__restrict__ z, double lox,
    double loy, double loz, double icx, double icy, double icz, int nx,
    int ny, int nz, uint32_t *__restrict__ bits) {
  for (size_t i = blockIdx.x * (size_t) blockDim.x + threadIdx.x; i < n;
       i += (size_t) gridDim.x * blockDim.x) {
    int cx = (int) floor((x[i] - lox) * icx);
    int cy = (int) floor((y[i] - loy) * icy);
    int cz = (int) floor((z[i] - loz) * icz);
    cx = cx < 0 ? 0 : (cx >= nx ? nx - 1 : cx);
    cy = cy < 0 ? 0 : (cy >= ny ? ny - 1 : cy);
    cz = cz < 0 ? 0 : (cz >= nz ? nz - 1 : cz);
    const size_t c = ((size_t) cz * ny + cy) * nx + cx;
    atomicOr(bits + (c >> 5), 1u << (c & 31));
  }
}

__global__ void k_popc(size_t nw, const uint32_t *__restrict__ bits,
    unsigned long long *count) {
  unsigned long long t = 0;
  for (size_t i = blockIdx.x * (size_t) blockDim.x + threadIdx.x; i < nw;
       i += (size_t) gridDim.x * blockDim.x)
    t += (unsigned long long) __popc(bits[i]);
  for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  if ((threadIdx.x & 31) == 0 && t) atomicAdd(count, t);
}

extern "C" int fcfcg_k_occupancy(void *stream, size_t n, const double *x,
    const double *y, const double *z, const double lo[3], const int dim[3],
    const double inv_cell[3], uint32_t *bits, size_t nw,
    unsigned long long *count) {
  cudaStream_t st = (cudaStream_t) stream;
  cudaError_t e = cudaMemsetAsync(bits, 0, sizeof(uint32_t) * nw, st);
  if (!e) e = cudaMemsetAsync(count, 0, sizeof(unsigned long long), st);
  if (e) return (int) e;
  if (n) {
    k_occupy<<<grid_for(n, PREP_THREADS), PREP_THREADS, 0, st>>>(
        n, x, y, z, lo[0], lo[1], lo[2], inv_cell[0], inv_cell[1],
        inv_cell[2], dim[0], dim[1], dim[2], bits);
    if ((e = cudaGetLastError())) return (int) e;
  }
  k_popc<<<grid_for(nw, PREP_THREADS), PREP_THREADS, 0, st>>>(nw, bits,
                                                               count);
  return (int) cudaGetLastError();
}

__global__ void k_unsort(size_t n, const uint32_t *__restrict__ sid,
    const double *__restrict__ in, double *__restrict__ out) {
  for (size_t p = blockIdx.x * (size_t) blockDim.x + threadIdx.x; p < n;
       p += (size_t) gridDim.x * blockDim.x)
    out[sid[p]] = in[p];
}

extern "C" int fcfcg_k_unsort(void *stream, size_t n, const uint32_t *sid,
    const double *in, double *out) {
  if (!n) return 0;
  k_unsort<<<grid_for(n, PREP_THREADS), PREP_THREADS, 0,
             (cudaStream_t) stream>>>(n, sid, in, out);
  return (int) cudaGetLastError();
}

extern "C" const char *fcfcg_cuda_errstr(int code) {
  return cudaGetErrorString((cudaError_t) code);
}

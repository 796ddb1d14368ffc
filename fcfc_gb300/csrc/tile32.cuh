/*
 * tile32.cuh -- the pair-counting kernel (instantiated by count32_*.cu): FP32
 * separations with an FP64 recheck, or (BIN_F64) every pair in FP64.
 *
 * Work decomposition (replaces FCFC's dual k-d tree, src/fcfc/2pt_box/
 * dual_tree.c:245-373, and its OpenMP/MPI node-pair scheduler,
 * count_func.c:7431-7722):
 *   - points are sorted into a coarse cell grid (cells about as wide as the
 *     largest separation that counts) and, inside a cell, along a Hilbert
 *     curve; a cell's points are cut into blocks of at most 32, each with
 *     its bounding box (prep.cu:k_runs);
 *   - the unit of work is a tile: the points of one block (A, in shared
 *     memory) against those of another (B, one per lane).  A persistent
 *     warp takes a block A from a global counter, tests the boxes of 32
 *     blocks B of the cell stencil at a time, one per lane, against A's and
 *     those of A's points by fours, and visits the tiles that can hold a
 *     pair, in each the fours that can (a surface of blocks of 32 around the
 *     outer range is 2.5 of its volume, of fours against blocks 2.06: 2e6
 *     points 24.6 -> 23.7 ms, log (s_perp, pi) of a survey 23.6 -> 22.6);
 *   - auto counts use half of the stencil, blocks from A's own on in A's
 *     cell, and i < j within a block.
 *
 * Warps share only the CTA's histogram: there is no barrier and no list in
 * the main loop (a batch has one per run of blocks of a catalogue).
 *
 * Per pair (FP32 path): separations on coordinates relative to the cell
 * centres, four points of A per step with packed FP32, the bin from the
 * separation itself (linear bins) or from a table of edges in shared
 * memory, and a rounding bound: a pair whose s^2, mu, s_perp^2 or pi lies
 * within the bound of a bin edge is queued and re-binned by the FP64 formula
 * of the reference (metric_common.c of src/fcfc/2pt_box and src/fcfc/2pt),
 * so integer counts equal the FP64 build.
 *
 * What bounds it: instruction issue and the FMA pipe (unweighted (s, mu)
 * mocks: issue slots 80 % used, FMA pipe 51 %, ALU 57 %; weighted: 75 %, with
 * 65 % of the shared wavefronts).  1.32 warp instructions per in-range pair
 * (weighted 2.52, survey 3.33), with 1.44 (1.44, 1.76) pairs tested for each in
 * range.  A kernel that tested candidates first, queued them and binned them
 * compacted took 2.8 (3.9, 4.8).  A pass before and after: (s, mu) box of 2e6
 * points weighted 33.6 -> 22.4 ms, (s_perp, pi) with log bins 6.4 -> 3.6, log
 * s bins of 4e5 points 3.9 -> 1.3, 256 mocks 631 -> 329, survey (s, mu) of 4e5
 * + 4e6 433 -> 299.
 *
 * Histograms live in shared memory (u32 counts, or int64 fixed-point weight
 * products) and are merged into global 64/128-bit integer accumulators, so
 * the results do not depend on the order of the additions.
 */
#ifndef FCFCG_TILE32_CUH
#define FCFCG_TILE32_CUH
#include "count_common.cuh"

/* 1 / sqrt(x): relative error <= 2^-22.9 (PTX ISA); 0 gives +inf. */
__device__ __forceinline__ float rsq_ftz(float x) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

/* Shared memory of a warp: its block A, four points' coordinates at a time;
 * 32 stencil entries; and its counters.  What the inner loop does not use is
 * kept here: its registers decide the CTAs per SM. */
struct TileWarp {
  ulonglong2 p[8][3];      /* points 4k .. 4k + 3: x, y, z of each */
  float4 gc[8], gh[8];     /* their boxes: centre, half extents */
  float4 sd[32];           /* stencil entry: -offset * width, image code */
  uint2 si[32];            /* its first block and their number */
  unsigned long long cnt[4];   /* as fcfcg_launch.stats */
  /* pairs to recheck, nrest of them: A's and B's index, image code and (from
   * bit 6) the catalogue */
  uint32_t ra[32], rb[32], rc[32], nrest, pad[3];
};
/* with weights: (round(w 2^30), remainder, w) of each point of A */
struct TileWarpW {
  TileWarp t;
  float4 aw[32];
};

/* adjoint: partial gradients of A's points, one word per lane and step (a
 * lane's is that of point 4 step + (lane & 3), over a quarter of the lanes) */
struct TileWarpA {
  TileWarpW w;
  long long ga[8][32];
};

/* all-FP64: pairs within the outer range, to be binned 32 at a time; and the
 * adjoint's FP64 gradients of A's points */
#define Q64 160
struct TileWarp64 {
  TileWarpW w;
  uint2 q[Q64];            /* sorted indices */
  uint8_t code[Q64];       /* image codes */
  double ga[32];
};

/* wt: 0 unweighted, 1 weighted, 2 adjoint, 3 all-FP64 */
__host__ __device__ __forceinline__ size_t tile_warp_bytes(int wt) {
  return wt == 3 ? sizeof(TileWarp64)
      : wt == 2 ? sizeof(TileWarpA)
                 : (wt ? sizeof(TileWarpW) : sizeof(TileWarp));
}

/* Two FP32 values in a 64-bit register, for the packed instructions: each
 * rounds its two components as the scalar ones do, in one issue slot (the
 * FMA pipe takes two cycles). */
typedef unsigned long long f2;
__device__ __forceinline__ f2 pack2(float a, float b) {
  f2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ f2 dup2(float a) {
  f2 r;
  asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(a));
  return r;
}
__device__ __forceinline__ float2 unpack2(f2 a) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(a));
  return r;
}
__device__ __forceinline__ f2 add2(f2 a, f2 b) {
  f2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 mul2(f2 a, f2 b) {
  f2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
  f2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

/* Add 1 to a 32-bit shared bin at a shared-space byte address where ok, and
 * to the lane's spare word elsewhere: a predicated shared atomic compiles to
 * a branch around it (3.3 branch instructions each).  (No memory clobber:
 * the bins are read only behind barriers and through atomics, and a clobber
 * has the launch parameters loaded again after each pair.) */
__device__ __forceinline__ void red_inc(uint32_t addr, uint32_t spare,
    bool ok) {
  asm volatile("red.shared.add.u32 [%0], 1;" :: "r"(ok ? addr : spare));
}

/* The same for a pair within the outer range (c) with no edge in its windows
 * (|f| < h, |fq| < hq); one with an edge sets bit BIT of rest.  The tests
 * chain through predicates. */
template <int BIT>
__device__ __forceinline__ void red_pair(uint32_t addr, uint32_t spare,
    bool in, float f, float h, float fq, float hq, uint32_t &rest) {
  asm volatile("{.reg .pred c, g, a, b; .reg .f32 t; .reg .u32 x;\n\t"
               "setp.ne.u32 c, %2, 0;\n\t"
               "abs.f32 t, %3; setp.lt.and.f32 g|a, t, %4, c;\n\t"
               "abs.f32 t, %5; setp.lt.and.f32 g|b, t, %6, g;\n\t"
               "@a or.b32 %0, %0, %7;\n\t"
               "@b or.b32 %0, %0, %7;\n\t"
               "selp.u32 x, %1, %8, g;\n\t"
               "red.shared.add.u32 [x], 1;}"
               : "+r"(rest) : "r"(addr), "r"((uint32_t) in), "f"(f), "f"(h),
                 "f"(fq), "f"(hq), "n"(BIT), "r"(spare));
}
template <int BIT>
__device__ __forceinline__ void red_pair(uint32_t addr, uint32_t spare,
    bool in, float f, float h, uint32_t &rest) {
  asm volatile("{.reg .pred c, g, a; .reg .f32 t; .reg .u32 x;\n\t"
               "setp.ne.u32 c, %2, 0;\n\t"
               "abs.f32 t, %3; setp.lt.and.f32 g|a, t, %4, c;\n\t"
               "@a or.b32 %0, %0, %5;\n\t"
               "selp.u32 x, %1, %6, g;\n\t"
               "red.shared.add.u32 [x], 1;}"
               : "+r"(rest) : "r"(addr), "r"((uint32_t) in), "f"(f), "f"(h),
                 "n"(BIT), "r"(spare));
}

/* Launch parameters of the inner loop, held in registers: as operands of
 * the constant bank two in one instruction cost a load each time. */
__device__ __forceinline__ float pin(float a) {
  asm volatile("" : "+f"(a));
  return a;
}
__device__ __forceinline__ uint32_t pin(uint32_t a) {
  asm volatile("" : "+r"(a));
  return a;
}
/* Weighted s histograms are held in 2^hlog copies, a lane's by its number: an
 * atomic that returns takes a turn per lane on the same word, and the lanes'
 * separations from one point lie in a bin or two (5.6e5 points, 23 bins: 2.26 ->
 * 1.58 ms a pass; (s, mu) bins of 4 copies gained nothing). */
#define HREP(WT, ADJ, B) ((WT) && !(ADJ) && IS_ISO(B))
struct LinConst {
  float slim;              /* the outer range */
  float inv, s0, hs;       /* linear s bins */
  float q0, nmu, q1, qc;   /* mu */
  float p0, pinv, hp;      /* linear pi bins */
  float ea, eb;            /* window of a table's value: ea s^2 + eb */
  float hc;                /* columns of a row */
  uint32_t ha, spare, hm;  /* shared bins: base, the lane's spare, bytes each */
};

/* An axis by table: cells of the value's FP32 bits >> lg from off on, the
 * last of n taking all below; (edge, 1.5 2^23 + column below the edge). */
struct EdgeTab {
  const float2 *t;
  int lg, off;
  uint32_t last;
};

#define TMAGIC 12582912.f                  /* 1.5 2^23 */
#define TMAGIC_BITS 0x4B400000u

/* Shared bin x (hcols columns per row, the first bin at row hrow0, column
 * hcol0) to the global bin, or -1 out of range. */
__device__ __forceinline__ int tile_gbin(const fcfcg_launch &L, uint32_t x) {
  const int s = (int) (x % (uint32_t) L.hcols) - L.hcol0;
  const int q = (int) (x / (uint32_t) L.hcols) - L.hrow0;
  if (s < 0 || s >= L.ns || q < 0 || q >= L.hrows) return -1;
  return s + q * L.ns;
}

/* fix_prod with the rounding constant and the cross term added before the
 * one shift: (p + 2^8 + 2^9 c) >> 9 = ((p + 2^8) >> 9) + c, the same integer
 * in fewer operations. */
__device__ __forceinline__ long long tile_prod(int ia, float ra, float fa,
    int ib, float rb, float fb) {
  const float c = __fadd_rn(__fmul_rn(fa, rb), __fmul_rn(ra, fb));
  const float t = __fmaf_rn(c, 2251799813685248.0f /* 2^51 */, TMAGIC);
  const long long p = (long long) ia * (long long) ib +
      (256ll - ((long long) TMAGIC_BITS << 9));
  return (p + (long long) __float_as_int(t) * 512ll) >> 9;
}

/*
 * Adjoint: the product of a weight and a cotangent entry, both scaled to at
 * most 1, in units of 2^-52: the integer parts (round(x 2^30)) multiply exactly
 * and are rounded by a shift, the cross terms with the remainders (weight's: ra,
 * scaled by 2^-30; entry's: rb), at most 2^-30 in sum, by the 1.5 2^23 trick (at
 * most 2^22 of them), and the product of the remainders (2^-10 of a unit) is left
 * out.  Within 1/2 + 1/2 unit and the cross terms' FP32 roundings (the two
 * remainders', the two factors', the product's and the sum's: at most 7/16
 * unit): 1.44; over 4e7 products the worst was 1.29, and the mean 0, also for
 * weights of 1, whose products have no low bits: with the sum of both rounded
 * once to whole units, the cross terms' halves all go up (0.14 units a product,
 * 10 times the error of a gradient of 5e5 terms).  An FP64 multiply-add per
 * product kept the FP64 pipe the bound (32 cycles of an SM per pair of a warp;
 * GB300 has 2 FP64 lanes per SM), at an error of up to 2 of these units.
 */
__device__ __forceinline__ long long adj_prod(int ia, float ra, float fa,
    int ib, float rb, float ib_f) {
  const float c = __fmaf_rn(fa, rb, __fmul_rn(ra, ib_f));
  const float t = __fmaf_rn(c, 4503599627370496.0f /* 2^52 */, TMAGIC);
  const long long p = (long long) ia * (long long) ib +
      (128ll - ((long long) TMAGIC_BITS << 8));
  return (p + (long long) __float_as_int(t) * 256ll) >> 8;
}

__device__ __forceinline__ long long shfl_xor64(long long v, int o) {
  const uint32_t lo = __shfl_xor_sync(FULLMASK, (uint32_t) v, o),
                 hi = __shfl_xor_sync(FULLMASK, (uint32_t) (v >> 32), o);
  return (long long) (((unsigned long long) hi << 32) | lo);
}

/* Four values per lane to one: lane l gets the sum of value l & 3 over the
 * lanes that differ from it in the low two bits. */
__device__ __forceinline__ long long reduce4(const long long v[4], int lane) {
  const bool b0 = lane & 1, b1 = lane & 2;
  long long r[2];
#pragma unroll
  for (int i = 0; i < 2; i++)
    r[i] = (b0 ? v[2 * i + 1] : v[2 * i]) +
           shfl_xor64(b0 ? v[2 * i] : v[2 * i + 1], 1);
  return (b1 ? r[1] : r[0]) + shfl_xor64(b1 ? r[0] : r[1], 2);
}

/* Add A's gradients (of at most 127 tiles) to the global ones and clear them. */
__device__ __forceinline__ void adj_flush(const fcfcg_launch &L, TileWarpA *S,
    uint32_t first, int m) {
  const int lane = threadIdx.x & 31;
  __syncwarp();
  /* (two sums: all eight words can pass 2^63) */
  long long v = 0, u = 0;
  for (int i = 0; i < 4; i++) {
    v += S->ga[lane >> 2][(lane & 3) + 4 * i];
    u += S->ga[lane >> 2][(lane & 3) + 16 + 4 * i];
  }
  if (lane < m && (v || u))
    atomicAdd(L.dA + first + lane, ((double) v + (double) u) * L.gunitA);
  __syncwarp();
  for (int i = 0; i < 8; i++) S->ga[i][lane] = 0;
  __syncwarp();
}

/* Weighted sums in shared memory: two 32-bit words per bin (the high words
 * hwords + 32 words behind), value = hi 2^32 + lo, lo unsigned and hi signed.
 * The carry out of lo is read from the returned value.  An add that finds hi
 * beyond +-2^30 takes all of hi by an exchange and adds it to the global 128-bit
 * accumulator: whatever the other threads do meanwhile, what is in the word is
 * counted once, and the adds under way (two of each of 256 threads, of 2^19 + 1
 * at most) do not carry it to 2^31.  Of a thread's two words the larger is taken;
 * the other, if beyond too, by the next add that finds it so: to rise a step (of
 * 2^19) further unseen it has to meet a larger one that is then cleared, which
 * doubles with each step.
 * (Moving 2^30 out at each step over the limit lost sums of mixed signs, of which
 * a warp's 32 adds to one word step over it several times before the first move
 * takes effect.  Carrying hi's own overflow took the sum too: weighted (s, mu) of
 * 2e6 points 23.4 ms a pass, 22.7 so; survey (s, mu) 311.7 and 300.7; exchanging
 * both words 22.3 and 305.4.) */
__device__ __forceinline__ uint32_t add_lo(uint32_t addr, uint32_t v) {
  uint32_t old;
  asm volatile("atom.shared.add.u32 %0, [%1], %2;"
               : "=r"(old) : "r"(addr), "r"(v));
  return old;
}
__device__ __forceinline__ int add_hi(uint32_t addr, int v) {
  int old;
  asm volatile("atom.shared.add.s32 %0, [%1], %2;"
               : "=r"(old) : "r"(addr), "r"(v));
  return old;
}
#define HI_LIMIT 0x40000000u
__device__ __forceinline__ void hi_out(const fcfcg_launch &L, uint32_t mock,
    uint32_t addr, uint32_t ah, uint32_t hb) {
  int v;
  asm volatile("atom.shared.exch.b32 %0, [%1], 0;" : "=r"(v) : "r"(ah));
  const int b = tile_gbin(L, (addr - hb) >> (2 + L.hlog));
  if (b >= 0)
    add128((L.mocks ? L.mocks[mock].gwt : L.gwt) + 2 * b,
           (long long) v * (1ll << 32));
}
/* Two weighted pairs: their atomics overlap. */
__device__ __forceinline__ void tile_add_w2(const fcfcg_launch &L,
    uint32_t mock, uint32_t hb, uint32_t a0, uint32_t a1, long long v0,
    long long v1) {
  const uint32_t ho = 4u * (uint32_t) ((L.hist_smem ? L.hwords : 0) + 32);
  const uint32_t l0 = add_lo(a0, (uint32_t) v0), l1 = add_lo(a1, (uint32_t) v1);
  const int h0 = (int) (v0 >> 32) + ((l0 + (uint32_t) v0) < l0 ? 1 : 0),
            h1 = (int) (v1 >> 32) + ((l1 + (uint32_t) v1) < l1 ? 1 : 0);
  const int o0 = add_hi(a0 + ho, h0), o1 = add_hi(a1 + ho, h1);
  if ((int) (((uint32_t) o0 + HI_LIMIT) | ((uint32_t) o1 + HI_LIMIT)) < 0 &&
      L.hist_smem) {
    const uint32_t a = abs(o1) > abs(o0) ? a1 : a0;
    hi_out(L, mock, a, a + ho, hb);
  }
}

/* State of a warp's tile. */
struct Tile {
  int m;                    /* points of A */
  uint32_t gm;              /* groups of four that can hold a pair */
  int ilim;                 /* this lane's pairs: A points below ilim */
  uint32_t first;           /* first sorted index of A */
  uint32_t bj;              /* this lane's sorted index */
  uint32_t code, mock;      /* image code of the cell pair, catalogue */
  float bx, by, bz;         /* this lane's point, from A's cell centre */
  float vx, vy, vz;         /* survey: 2 b + 2 c_A */
  float ux, uy, uz, lh, lP; /* survey (s_perp, pi): line-of-sight cut */
  int wi;                   /* this lane's weight */
  float wr, wf;
};

/* Column of a value in a table, as 1.5 2^23 + column: the cell's, plus one
 * from the cell's edge on; the edge's distance goes to dist.  A cell with
 * several edges near it holds a NaN: the distance then exceeds no window. */
__device__ __forceinline__ float tab_col(const EdgeTab &E, float v,
    float &dist) {
  const uint32_t i = (__float_as_uint(v) >> E.lg) - (uint32_t) E.off;
  const float2 e = E.t[i < E.last ? i : E.last];
  const float d = __fsub_rn(v, e.x);
  dist = fabsf(d);
  return d >= 0.f ? __fadd_rn(e.y, 1.f) : e.y;
}

/*
 * The bins of two pairs.
 *
 * Linear bins: t = (s + s0) inv rounds to the bin's column rn(t) by adding
 * 1.5 2^23 (no conversion instruction), and an edge lies within the window W
 * of t when |t - rn(t)| >= 1/2 - W; W is taken at the top of the range.  mu
 * likewise with t = (mu + q0) nmu, its window's term in q at q = nmu, so
 * that one FMA remains; linear pi bins likewise.  Other bins: the edge table
 * (tab_col) of s^2, s_perp^2 or pi (survey: pi^2), the window a linear bound
 * ea s^2 + eb.
 *
 * v: 1.5 2^23 + the shared bin (row hcols + column, exact below 2^22), so that
 * its low bits are the bin.  No edge lies within the windows when |f| < h and |g| <
 * k (k = 1, g = 0 without a second axis).
 */
struct PairBin {
  f2 v, f, h, g, k;
  f2 col, nq;              /* 1.5 2^23 + column; - row */
  f2 s;                    /* s^2 or s_perp^2 */
  float2 pi;
};
template <int GEOM, int BIN>
__device__ __forceinline__ PairBin pair_bin(const LinConst &C,
    const EdgeTab &ES, const EdgeTab &EP, f2 s2p, f2 dzp, f2 dmp, f2 mmp) {
  constexpr bool SURVEY = GEOM == FCFCG_GEOM_SURVEY;
  PairBin p;
  const f2 mag = dup2(TMAGIC), neg = dup2(-1.f);
  const float2 s2 = unpack2(s2p);
  f2 rs = 0;
  if (LINS(BIN) || IS_SMU(BIN)) rs = pack2(rsq_ftz(s2.x), rsq_ftz(s2.y));
  /* rows: mu or pi */
  f2 nq = 0;                        /* - the row */
  f2 sv = s2p;                      /* the s axis' value */
  if (IS_SMU(BIN)) {
    f2 x;
    if (SURVEY) {
      const float2 m = unpack2(mul2(mmp, s2p)), d = unpack2(dmp);
      x = pack2(fabsf(d.x) * rsq_ftz(m.x), fabsf(d.y) * rsq_ftz(m.y));
    } else {
      const float2 d = unpack2(dzp), q = unpack2(rs);
      x = pack2(fabsf(d.x) * q.x, fabsf(d.y) * q.y);
    }
    const f2 q = add2(x, dup2(C.q0)), nmu = dup2(C.nmu);
    nq = fma2(fma2(q, nmu, mag), neg, mag);
    p.g = fma2(q, nmu, nq);
    p.k = fma2(dup2(C.q1), rs, dup2(C.qc));
  } else if (IS_SPI(BIN)) {
    float2 &pi = p.pi;
    if (SURVEY) {
      /* pi = |d.m| / |m|, s_perp^2 = s^2 - pi^2 */
      const float2 m = unpack2(mmp), d = unpack2(dmp);
      pi = make_float2(fabsf(d.x) * rsq_ftz(m.x), fabsf(d.y) * rsq_ftz(m.y));
      const f2 pp = pack2(pi.x, pi.y);
      sv = fma2(mul2(pp, neg), pp, s2p);
    } else {
      const float2 d = unpack2(dzp);
      pi = make_float2(fabsf(d.x), fabsf(d.y));
    }
    if (LINP(BIN)) {
      const f2 q = add2(pack2(pi.x, pi.y), dup2(C.p0)), inv = dup2(C.pinv);
      nq = fma2(fma2(q, inv, mag), neg, mag);
      p.g = fma2(q, inv, nq);
      p.k = dup2(C.hp);
    } else {
      float dx, dy;
      const float rx = tab_col(EP, pi.x, dx), ry = tab_col(EP, pi.y, dy);
      nq = fma2(pack2(rx, ry), neg, mag);
      p.g = dup2(C.hp);
      p.k = pack2(dx, dy);
    }
  } else {
    p.g = 0;
    p.k = dup2(1.f);
  }
  /* columns: s or s_perp */
  f2 col;
  if (LINS(BIN)) {
    const f2 s = fma2(s2p, rs, dup2(C.s0)), inv = dup2(C.inv);
    col = fma2(s, inv, mag);
    p.f = fma2(s, inv, fma2(col, neg, mag));
    p.h = dup2(C.hs);
  } else {
    const float2 v = unpack2(sv);
    float dx, dy;
    const float cx = tab_col(ES, v.x, dx), cy = tab_col(ES, v.y, dy);
    col = pack2(cx, cy);
    p.f = fma2(s2p, dup2(C.ea), dup2(C.eb));
    p.h = pack2(dx, dy);
  }
  p.v = IS_ISO(BIN) ? col : fma2(nq, dup2(-C.hc), col);
  p.col = col;
  p.s = sv;
  p.nq = nq;
  return p;
}

/* The bin's word of a pair of pair_bin, in integers: p.v holds it in a float,
 * exact below 2^22, which shared bins are and the adjoint's table in global
 * memory may not be. */
__device__ __forceinline__ uint32_t tile_word(const PairBin &p, int e,
    int hcols) {
  const float2 c = unpack2(p.col), q = unpack2(p.nq);
  return __float_as_uint(e ? c.y : c.x) - TMAGIC_BITS +
         (uint32_t) -(e ? q.y : q.x) * (uint32_t) hcols;
}

__device__ __forceinline__ LinConst lin_const(const fcfcg_launch &L) {
  LinConst C;
  C.slim = L.s_lim;
  C.inv = L.tl_inv;
  C.s0 = L.tl_s0;
  C.hs = L.tl_h;
  C.q0 = L.tl_q0;
  C.nmu = L.fnmu;
  C.q1 = -L.tl_q1;
  C.qc = L.tl_qc;
  C.p0 = L.tl_p0;
  C.pinv = L.tl_pinv;
  C.hp = L.tl_hp;
  C.ea = L.tl_ea;
  C.eb = L.tl_eb;
  C.hc = (float) L.hcols;
  C.ha = C.spare = C.hm = 0;
  return C;
}

/*
 * Without a shared histogram: the pairs of a tile (mask: this lane's) into
 * the global one, by FP32 where the windows allow; the others are returned.
 * A lane takes its points of A two at a time, and unweighted additions return
 * nothing (1e5 points, 8e4 bins: 3.66 ms with the generic atomic, 2.47 with red;
 * with two points the same for all lanes 2.67).
 */
template <int GEOM, int BIN, int WT>
__device__ __noinline__ uint32_t tile_global(const fcfcg_launch &L,
    const Tile T, TileWarpW *S, uint32_t mask, const EdgeTab ES,
    const EdgeTab EP) {
  const fcfcg_mock *M = L.mocks ? L.mocks + T.mock : NULL;
  unsigned long long *out = WT ? (M ? M->gwt : L.gwt) : (M ? M->gcnt : L.gcnt);
  const LinConst C = lin_const(L);
  const f2 nbx = dup2(-T.bx), nby = dup2(-T.by), nbz = dup2(-T.bz);
  uint32_t n_in = 0;
  uint32_t left = mask;
  mask = 0;
  while (left) {
    /* two points of A (the last one alone) */
    const int i0 = __ffs((int) left) - 1;
    left &= left - 1u;
    const bool two = left != 0u;
    const int i1 = two ? __ffs((int) left) - 1 : i0;
    left &= left - 1u;
    const float *a = (const float *) S->t.p[i0 >> 2] + (i0 & 3),
                *b = (const float *) S->t.p[i1 >> 2] + (i1 & 3);
    const f2 dx = add2(pack2(a[0], b[0]), nbx), dy = add2(pack2(a[4], b[4]), nby),
             dz = add2(pack2(a[8], b[8]), nbz);
    f2 s2 = fma2(dy, dy, mul2(dx, dx)), dm = 0, mm = 0;
    if (!IS_SPI(BIN) || GEOM == FCFCG_GEOM_SURVEY) s2 = fma2(dz, dz, s2);
    if (GEOM == FCFCG_GEOM_SURVEY) {
      const f2 mx = add2(dup2(T.vx), dx), my = add2(dup2(T.vy), dy),
               mz = add2(dup2(T.vz), dz);
      dm = fma2(dz, mz, fma2(dy, my, mul2(dx, mx)));
      mm = fma2(mz, mz, fma2(my, my, mul2(mx, mx)));
    }
    const PairBin p = pair_bin<GEOM, BIN>(C, ES, EP, s2, dz, dm, mm);
    const float2 f = unpack2(p.f), fh = unpack2(p.h), g = unpack2(p.g),
                 gk = unpack2(p.k), mm2 = unpack2(mm), col = unpack2(p.col),
                 nq = unpack2(p.nq);
#pragma unroll
    for (int e = 0; e < 2; e++) {
      if (e && !two) break;
      const int i = e ? i1 : i0;
      const float m = e ? mm2.y : mm2.x;
      bool plain = (fabsf(e ? f.y : f.x) < (e ? fh.y : fh.x)) &
                   (fabsf(e ? g.y : g.x) < (e ? gk.y : gk.x));
      if (GEOM == FCFCG_GEOM_SURVEY && !IS_ISO(BIN)) plain &= m >= L.m2min;
      /* (next to the observer pi's error is not bounded: rechecked) */
      if (GEOM == FCFCG_GEOM_SURVEY && IS_SPI(BIN) && m >= L.m2min &&
          !((e ? p.pi.y : p.pi.x) < L.p_lim))
        continue;
      if (!plain) {
        mask |= 1u << i;
        continue;
      }
      const int s = (int) (__float_as_uint(e ? col.y : col.x) - TMAGIC_BITS) -
                    L.hcol0,
                q = (int) -(e ? nq.y : nq.x) - L.hrow0;
      if (s < 0 || s >= L.ns || q < 0 || q >= L.hrows) continue;
      const int bin = s + q * L.ns;
      n_in++;
      if (WT) {
        const float4 wa = S->aw[i];
        add128(out + 2 * bin,
               fix_prod(__float_as_int(wa.x), wa.y, wa.z, T.wi, T.wr, T.wf));
      } else {
        asm volatile("red.global.add.u64 [%0], 1;"
                     :: "l"(__cvta_generic_to_global(out + bin)) : "memory");
      }
    }
  }
  __syncwarp();
  n_in = __reduce_add_sync(FULLMASK, n_in);
  if ((threadIdx.x & 31) == 0) S->t.cnt[1] += n_in;
  __syncwarp();
  return mask;
}

/* A pair by the FP64 formula where the queue is full: is it in range? */
template <int WT, int ADJ>
__device__ __forceinline__ uint32_t rest_bin(const fcfcg_launch &L, uint32_t a,
    uint32_t b, uint32_t c) {
  const fcfcg_mock *M = L.mocks ? L.mocks + (c >> 6) : NULL;
  const int bin = ref_bin_pair(L, a, b, c & 63u, M ? M->box : L.box);
  if (bin < 0) return 0u;
  if (ADJ) adj_pair(L, a, b, bin);
  else if (WT) add128((M ? M->gwt : L.gwt) + 2 * bin, fix_prod_pair(L, a, b));
  else atomicAdd((M ? M->gcnt : L.gcnt) + bin, 1ull);
  return 1u;
}

/*
 * The collected pairs, and those of a tile that are left (bit i of rest: this
 * lane's point and A's i), to the FP64 recheck queue -- the warp reserves their
 * places with one atomic, whose answer it waits for: where the observer is
 * inside a survey tiles leave hundreds of pairs each (3e4 points around it,
 * (s, mu): 0.69 ms 32 at a time, 0.31 so).  Those beyond the queue's capacity
 * are binned here by the FP64 formula.  Every pair counts in the queue's 64-bit
 * fill counter, queued or not, so the counter cannot wrap and hand out slots
 * twice.
 */
template <int WT, int ADJ>
__device__ __noinline__ void rest_flush(const fcfcg_launch &L, TileWarp *t,
    uint32_t rest, uint32_t first, uint32_t bj, uint32_t code) {
  const int lane = threadIdx.x & 31;
  __syncwarp();
  const uint32_t n = t->nrest, own = (uint32_t) __popc(rest);
  uint32_t upto = own;
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t v = __shfl_up_sync(FULLMASK, upto, o);
    if (lane >= o) upto += v;
  }
  const uint32_t total = n + __shfl_sync(FULLMASK, upto, 31);
  unsigned long long slot = 0;
  if (lane == 0 && total) slot = atomicAdd(L.qcount, (unsigned long long) total);
  slot = __shfl_sync(FULLMASK, slot, 0);
  uint32_t n_in = 0, n_inl = 0;
  if ((uint32_t) lane < n) {
    const uint32_t a = t->ra[lane], b = t->rb[lane], c = t->rc[lane];
    if (slot + lane < L.qcap) {
      ((uint4 *) L.queue)[slot + lane] = make_uint4(a, b, c & 63u, c >> 6);
    } else {
      n_inl++;
      n_in += rest_bin<WT, ADJ>(L, a, b, c);
    }
  }
  for (slot += n + upto - own; rest; slot++) {
    const uint32_t a = first + (uint32_t) (__ffs((int) rest) - 1);
    rest &= rest - 1u;
    if (slot < L.qcap) {
      ((uint4 *) L.queue)[slot] = make_uint4(a, bj, code & 63u, code >> 6);
    } else {
      n_inl++;
      n_in += rest_bin<WT, ADJ>(L, a, bj, code);
    }
  }
  __syncwarp();
  n_in = __reduce_add_sync(FULLMASK, n_in);
  n_inl = __reduce_add_sync(FULLMASK, n_inl);
  if (lane == 0) {
    t->cnt[1] += n_in;
    t->cnt[2] += total;
    t->cnt[3] += n_inl;
    t->nrest = 0;
  }
  __syncwarp();
}

/* Collect the pairs a tile left (bit i of rest: this lane's point and A's i).
 * Every second tile has one or two: they go to the queue 32 at a time, whose
 * atomic and writes took a tile's turn 150 instructions otherwise. */
template <int WT, int ADJ>
__device__ __forceinline__ void tile_rest(const fcfcg_launch &L, TileWarp *t,
    uint32_t rest, uint32_t first, uint32_t bj, uint32_t code) {
  const uint32_t below = (1u << (threadIdx.x & 31)) - 1u;
  uint32_t bal;
  while ((bal = __ballot_sync(FULLMASK, rest != 0u)) != 0u) {
    const uint32_t n = (uint32_t) __popc(bal);
    if (t->nrest + n > 32u) {
      rest_flush<WT, ADJ>(L, t, rest, first, bj, code);
      break;
    }
    const uint32_t at = t->nrest + (uint32_t) __popc(bal & below);
    if (rest) {
      t->ra[at] = first + (uint32_t) (__ffs((int) rest) - 1);
      t->rb[at] = bj;
      t->rc[at] = code;
      rest &= rest - 1u;
    }
    __syncwarp();
    if ((threadIdx.x & 31) == 0) t->nrest += n;
    __syncwarp();
  }
}

template <int WT, int ADJ>
__device__ __noinline__ void tile_rest_call(const fcfcg_launch &L,
    TileWarp *t, uint32_t rest, uint32_t first, uint32_t bj, uint32_t code) {
  tile_rest<WT, ADJ>(L, t, rest, first, bj, code);
}

/*
 * The pairs of one tile: this lane's point against every point of A, four
 * at a time with packed FP32.  A step none of whose pairs is within the
 * outer range ends after the distance test.  Returns the pairs left for
 * tile_rest.
 *
 * The columns and rows around the bins (hcol0, hrow0 before the first and
 * one after the last) take the pairs out of range and are dropped when the
 * histogram is handed over, so no pair is tested against the range's ends.
 * s^2 near zero needs no test: tl_q1 makes the mu test fail there
 * (ctx.c:tile_bounds), and without mu a separation's error is bounded for
 * every s.
 *
 * SP: pairs i >= ilim are left out (blocks meeting themselves) and, for
 * surveys, the line of sight is tested for pairs next to the observer; the
 * plain variant is for the other tiles.
 */
template <int GEOM, int BIN, int WT, int ADJ, bool SP>
__device__ __forceinline__ uint32_t tile_pairs(const fcfcg_launch &L,
    const LinConst &C, const Tile &T, TileWarpW *S, uint32_t hb,
    const EdgeTab &ES, const EdgeTab &EP, uint32_t &n_in, long long &gb) {
  constexpr bool SURVEY = GEOM == FCFCG_GEOM_SURVEY;
  constexpr bool TWO = !IS_ISO(BIN);     /* a second axis */
  constexpr bool LOS = SURVEY && !IS_ISO(BIN), CUT = LOSCUT(GEOM, BIN);
  const f2 nbx = dup2(-T.bx), nby = dup2(-T.by), nbz = dup2(-T.bz);
  uint32_t rest = 0;
#pragma unroll 1
  for (uint32_t gm = T.gm; gm; gm &= gm - 1u) {
    const int q = __ffs((int) gm) - 1, k = 4 * q;
    const ulonglong2 X = S->t.p[q][0], Y = S->t.p[q][1], Z = S->t.p[q][2];
    const f2 dx[2] = {add2(X.x, nbx), add2(X.y, nbx)};
    const f2 dy[2] = {add2(Y.x, nby), add2(Y.y, nby)};
    const f2 dz[2] = {add2(Z.x, nbz), add2(Z.y, nbz)};
    f2 s2[2];
    bool c[4];
#pragma unroll
    for (int h = 0; h < 2; h++) {
      s2[h] = fma2(dy[h], dy[h], mul2(dx[h], dx[h]));
      if (IS_SPI(BIN) && !SURVEY) {
        const float2 v = unpack2(s2[h]), z = unpack2(dz[h]);
        c[2 * h] = (fabsf(z.x) < L.p_lim) & (v.x < L.s_lim);
        c[2 * h + 1] = (fabsf(z.y) < L.p_lim) & (v.y < L.s_lim);
      } else {
        s2[h] = fma2(dz[h], dz[h], s2[h]);
        const float2 v = unpack2(s2[h]);
        c[2 * h] = v.x < C.slim;
        c[2 * h + 1] = v.y < C.slim;
        if (CUT) {
          /* not beyond pi_max for sure */
          const float2 t = unpack2(fma2(dz[h], dup2(T.uz),
              fma2(dy[h], dup2(T.uy), mul2(dx[h], dup2(T.ux)))));
          const float2 r = unpack2(fma2(s2[h], dup2(T.lh), dup2(T.lP)));
          c[2 * h] = c[2 * h] & (fabsf(t.x) < r.x);
          c[2 * h + 1] = c[2 * h + 1] & (fabsf(t.y) < r.y);
        }
      }
      if (SP) {
        c[2 * h] = c[2 * h] & (k + 2 * h < T.ilim);
        c[2 * h + 1] = c[2 * h + 1] & (k + 2 * h + 1 < T.ilim);
      }
    }
    if (!__ballot_sync(FULLMASK, (c[0] | c[1]) | (c[2] | c[3]))) continue;
    uint32_t r4 = 0;
    long long ga[4];          /* adjoint: terms of A's four points */
#pragma unroll
    for (int h = 0; h < 2; h++) {
      f2 dm = 0, mm = 0;
      if (LOS) {
        /* line of sight m = x_a + x_b = (2 b + 2 c_A) + d */
        const f2 mx = add2(dup2(T.vx), dx[h]), my = add2(dup2(T.vy), dy[h]),
                 mz = add2(dup2(T.vz), dz[h]);
        dm = fma2(dz[h], mz, fma2(dy[h], my, mul2(dx[h], mx)));
        mm = fma2(mz, mz, fma2(my, my, mul2(mx, mx)));
      }
      const PairBin p = pair_bin<GEOM, BIN>(C, ES, EP, s2[h], dz[h], dm, mm);
      const float2 v = unpack2(p.v), f = unpack2(p.f), fh = unpack2(p.h),
                   g = unpack2(p.g), gk = unpack2(p.k), mm2 = unpack2(mm);
      uint32_t wat[2];        /* weighted pairs: their bins' addresses */
#pragma unroll
      for (int e = 0; e < 2; e++) {
        bool in = c[2 * h + e];
        if (SURVEY && IS_SPI(BIN)) {
          /* (next to the observer pi's error is not bounded: rechecked) */
          bool cut = (e ? p.pi.y : p.pi.x) < L.p_lim;
          if (SP) cut = cut | ((e ? mm2.y : mm2.x) < L.m2min);
          in = in & cut;
        }
        /* the shared bin's byte address */
        const uint32_t at = __float_as_uint(e ? v.y : v.x) *
                            (HREP(WT, ADJ, BIN) ? C.hm : 4u) + C.ha;
        const float fe = e ? f.y : f.x,
                    he = LINS(BIN) ? C.hs : (e ? fh.y : fh.x),
                    ge = IS_SPI(BIN) && !LINP(BIN) ? C.hp : (e ? g.y : g.x),
                    ke = LINP(BIN) ? C.hp : (e ? gk.y : gk.x);
        if (!WT && !SP) {
          if (TWO) {
            if (h == 0 && e == 0) red_pair<1>(at, C.spare, in, fe, he, ge, ke, r4);
            if (h == 0 && e == 1) red_pair<2>(at, C.spare, in, fe, he, ge, ke, r4);
            if (h == 1 && e == 0) red_pair<4>(at, C.spare, in, fe, he, ge, ke, r4);
            if (h == 1 && e == 1) red_pair<8>(at, C.spare, in, fe, he, ge, ke, r4);
          } else {
            if (h == 0 && e == 0) red_pair<1>(at, C.spare, in, fe, he, r4);
            if (h == 0 && e == 1) red_pair<2>(at, C.spare, in, fe, he, r4);
            if (h == 1 && e == 0) red_pair<4>(at, C.spare, in, fe, he, r4);
            if (h == 1 && e == 1) red_pair<8>(at, C.spare, in, fe, he, r4);
          }
          continue;
        }
        bool plain = fabsf(fe) < he;
        if (TWO) plain = plain & (fabsf(ge) < ke);
        if (LOS && SP) plain = plain & ((e ? mm2.y : mm2.x) >= L.m2min);
        const bool ok = in & plain;
        if (in & !plain) r4 |= 1u << (2 * h + e);
        if (!WT) {
          red_inc(at, C.spare, ok);
          continue;
        }
        /* counted as in range unless in a row or column around the bins
         * (above them, only a survey's s_perp can be) */
        const float2 s1 = unpack2(p.s);
        const float se = e ? s1.y : s1.x;
        bool inside = ok & (se >= L.tl_slo);
        if (IS_SPI(BIN)) {
          inside = inside & ((e ? p.pi.y : p.pi.x) >= L.tl_plo);
          if (SURVEY) inside = inside & (se < L.tl_shi);
        }
        n_in += (uint32_t) inside;
        wat[e] = ok ? at : C.spare;
      }
      if (ADJ) {
        /* d/dw_a of w_a w_b g[bin] is w_b g[bin], and the other way round;
         * spare and outer bins hold g = 0 */
#pragma unroll
        for (int e = 0; e < 2; e++) {
          int2 g;
          if (L.hist_smem)
            asm("ld.shared.v2.s32 {%0, %1}, [%2];"
                : "=r"(g.x), "=r"(g.y) : "r"(2u * wat[e] - hb));
          else
            g = __ldg((const int2 *) L.gtab +
                      (wat[e] == C.spare ? (wat[e] - hb) >> 2
                                         : tile_word(p, e, L.hcols)));
          const float4 wa = S->aw[k + 2 * h + e];
          const float gf = (float) g.x, gr = __int_as_float(g.y);
          ga[2 * h + e] = adj_prod(T.wi, T.wr, T.wf, g.x, gr, gf);
          gb += adj_prod(__float_as_int(wa.x), wa.y, wa.z, g.x, gr, gf);
        }
      } else if (WT) {
        const float4 w0 = S->aw[k + 2 * h], w1 = S->aw[k + 2 * h + 1];
        tile_add_w2(L, T.mock, hb, wat[0], wat[1],
                    tile_prod(__float_as_int(w0.x), w0.y, w0.z, T.wi, T.wr,
                              T.wf),
                    tile_prod(__float_as_int(w1.x), w1.y, w1.z, T.wi, T.wr,
                              T.wf));
      }
    }
    if (ADJ) {
      long long *acc = ((TileWarpA *) S)->ga[k >> 2];
      const int lane = threadIdx.x & 31;
      acc[lane] += reduce4(ga, lane);
    }
    rest |= r4 << k;
  }
  return rest;
}

/* The boxes of A's points by fours (as the blocks', prep.cu:k_runs); v: this
 * lane's point. */
__device__ __forceinline__ void group_box(TileWarp &t, const float4 &v,
    int lane, int m) {
  float mn[3] = {v.x, v.y, v.z}, mx[3] = {v.x, v.y, v.z};
  if (lane >= m)
    for (int d = 0; d < 3; d++) {
      mn[d] = 3e38f;
      mx[d] = -3e38f;
    }
#pragma unroll
  for (int o = 1; o < 4; o <<= 1)
#pragma unroll
    for (int d = 0; d < 3; d++) {
      mn[d] = fminf(mn[d], __shfl_xor_sync(FULLMASK, mn[d], o));
      mx[d] = fmaxf(mx[d], __shfl_xor_sync(FULLMASK, mx[d], o));
    }
  if (lane & 3) return;
  float c[3], h[3];
#pragma unroll
  for (int d = 0; d < 3; d++) {
    c[d] = 0.5f * mn[d] + 0.5f * mx[d];
    h[d] = __fmul_ru(fmaxf(__fsub_ru(mx[d], c[d]), __fsub_ru(c[d], mn[d])),
                     1.000001f);
    if (lane >= m) {           /* no points: far from everything */
      c[d] = 1e30f;
      h[d] = 0.f;
    }
  }
  t.gc[lane >> 2] = make_float4(c[0], c[1], c[2], 0.f);
  t.gh[lane >> 2] = make_float4(h[0], h[1], h[2], 0.f);
}

/*
 * Survey (s_perp, pi): are all pairs of two blocks beyond pi_max for sure?
 * For a = a0 + h_a, b = b0 + h_b the line of sight m = a + b is within |h|,
 * h = h_a + h_b, of m0 = a0 + b0, its direction within 1.05 |h| / |m0| of u0 =
 * m0 / |m0| where |h| < |m0| / 2, and
 *   pi = |d.m| / |m| >= |(a0 - b0).u0| - sum h_k |u0_k| - Rs 1.05 |h| / |m0|
 * for separations within the outer range Rs.  los_p holds a slack far above the
 * rounding where |m0| >= 2 R; nearer the observer u0 itself can be rounding
 * noise (of single points h = 0 and |m0| as small as you like), and the blocks
 * are kept.  The sphere alone lets in 1.6 times the tiles of a cylinder of
 * radius 100 and length 2 x 40.
 */
__device__ __forceinline__ bool los_apart(const fcfcg_launch &L, float c2x,
    float c2y, float c2z, const float4 &ac, const float4 &ah, float bx,
    float by, float bz, const float4 &bh) {
  const float mx = c2x + (ac.x + bx), my = c2y + (ac.y + by),
              mz = c2z + (ac.z + bz);
  const float hx = ah.x + bh.x, hy = ah.y + bh.y, hz = ah.z + bh.z;
  const float m2 = fmaf(mz, mz, fmaf(my, my, mx * mx)),
              h2 = fmaf(hz, hz, fmaf(hy, hy, hx * hx)), ir = rsq_ftz(m2);
  const float dm = fmaf(ac.z - bz, mz, fmaf(ac.y - by, my, (ac.x - bx) * mx));
  const float hm = fmaf(hz, fabsf(mz), fmaf(hy, fabsf(my), hx * fabsf(mx))) +
                   1.1f * sqrtf(h2 * L.los_r2min);
  return m2 >= L.m2min && h2 < 0.2f * m2 && (fabsf(dm) - hm) * ir >= L.los_p;
}

/* All-FP64: bin n <= 32 queued pairs by the reference's formula, every lane
 * busy. */
template <int WT>
__device__ __forceinline__ void bin64(const fcfcg_launch &L, TileWarp64 *S,
    uint32_t *h, int first, int n, uint32_t &n_in) {
  const int lane = threadIdx.x & 31;
  if (lane >= n) return;
  const uint2 e = S->q[first + lane];
  const int bin = ref_bin_pair(L, e.x, e.y, S->code[first + lane], L.box);
  if (bin < 0) return;
  if (WT) {
    n_in++;
    const double v = __dmul_rn(L.A.w[e.x], L.B.w[e.y]);
    if (L.hist_smem) atomicAdd((double *) h + bin, v);
    else atomicAdd(L.gwd + bin, v);
  } else if (L.hist_smem) {
    atomicAdd(h + bin, 1u);
  } else {
    n_in++;
    atomicAdd(L.gcnt + bin, 1ull);
  }
}

/*
 * The pairs of one tile in FP64.  The FP32 distances, with their rounding
 * bound, only leave out pairs beyond the outer range (half of a tile's are
 * within it, and an FP64 instruction takes an SM 16 cycles whether its lanes
 * are active or not); the others are collected and binned 32 at a time.  nq:
 * pairs collected.  The adjoint bins a point of A against the lanes' points
 * and sums its terms across them.
 *
 * Bound by the FP64 pipe (2 lanes per SM and clock): 8 operations per pair
 * for the separation, and few others since the mu bin is taken from FP32
 * where that is certain (ref_mu).  Weighted (s, mu) count of a box of 3e4
 * points, 2.6e7 pairs: 15.0 -> 1.7 ms against a kernel that took every pair
 * of the neighbouring cells, with an FP64 division each.
 */
template <int GEOM, int WT, int ADJ>
__device__ __forceinline__ void tile_pairs64(const fcfcg_launch &L,
    const Tile &T, TileWarp64 *S, uint32_t *h, int &nq, uint32_t &n_in) {
  const int lane = threadIdx.x & 31;
  const bool cyl = GEOM == FCFCG_GEOM_BOX && L.bintype == FCFCG_BIN_SPI;
  double gb = 0;
#pragma unroll 1
  for (uint32_t gm = T.gm; gm; gm &= gm - 1u) {
    const int k = 4 * (__ffs((int) gm) - 1);
    const float *P = (const float *) S->w.t.p[k >> 2];
#pragma unroll 1
    for (int e = 0; e < 4; e++) {
      const float dx = P[e] - T.bx, dy = P[4 + e] - T.by, dz = P[8 + e] - T.bz;
      float s2 = fmaf(dy, dy, dx * dx);
      if (!cyl) s2 = fmaf(dz, dz, s2);
      /* (an infinite limit keeps every pair) */
      const bool in = (k + e < T.ilim) & !(s2 > L.s_lim) &
                      (!cyl | !(fabsf(dz) > L.p_lim));
      const uint32_t bal = __ballot_sync(FULLMASK, in);
      if (!bal) continue;
      const uint32_t a = T.first + (uint32_t) (k + e);
      if (ADJ) {
        double va = 0;
        const int bin = in ? ref_bin_pair(L, a, T.bj, T.code, L.box) : -1;
        if (bin >= 0) {
          n_in++;
          const double g = __ldg(L.gadj + bin);
          va = __dmul_rn(L.B.w[T.bj], g);
          gb = __dadd_rn(gb, __dmul_rn(L.A.w[a], g));
        }
        for (int o = 16; o > 0; o >>= 1)
          va = __dadd_rn(va, __shfl_xor_sync(FULLMASK, va, o));
        if (lane == 0) S->ga[k + e] = __dadd_rn(S->ga[k + e], va);
        continue;
      }
      if (in) {
        const int q = nq + __popc(bal & ((1u << lane) - 1u));
        S->q[q] = make_uint2(a, T.bj);
        S->code[q] = (uint8_t) T.code;
      }
      nq += __popc(bal);
    }
    if (!ADJ && nq >= 32) {
      __syncwarp();
      int f = 0;
      for (; f + 32 <= nq; f += 32) bin64<WT>(L, S, h, f, 32, n_in);
      __syncwarp();
      if (f + lane < nq) {
        const uint2 q = S->q[f + lane];
        const uint8_t c = S->code[f + lane];
        S->q[lane] = q;
        S->code[lane] = c;
      }
      nq -= f;
      __syncwarp();
    }
  }
  if (ADJ && gb != 0.0) atomicAdd(L.dB + T.bj, gb);
}

/* Add the shared histogram to a global one and clear it, by threads t0,
 * t0 + nt, ... (whole warps); unweighted counts handed over are counted as
 * in range.  Exchanges, so that other warps may go on adding meanwhile. */
template <int WT, bool F64 = false>
__device__ __noinline__ void tile_handover(const fcfcg_launch &L,
    uint32_t *h, uint32_t mock, int t0, int nt, TileWarp *S) {
  if (WT && F64) {
    double *g = L.gwd + (size_t) (blockIdx.x % fcfcg_gwd_copies(L.ntot)) * L.ntot;
    for (int x = t0; x < L.hlen; x += nt) {
      const double v = ((double *) h)[x];
      if (v != 0) atomicAdd(g + x, v);
    }
    return;
  }
  unsigned long long *g = WT ? (L.mocks ? L.mocks[mock].gwt : L.gwt)
                             : (L.mocks ? L.mocks[mock].gcnt : L.gcnt);
  unsigned long long sum = 0;
  for (uint32_t x = (uint32_t) t0; x < (uint32_t) L.hwords; x += (uint32_t) nt) {
    const int b = tile_gbin(L, x >> L.hlog);
    if (WT) {
      const long long v = ((long long) ((int *) h)[L.hwords + 32 + x] << 32) +
                          (long long) h[x];
      h[x] = 0;
      h[L.hwords + 32 + x] = 0;
      if (v && b >= 0) add128(g + 2 * b, v);
    } else {
      const uint32_t v = atomicExch(h + x, 0u);
      if (v && b >= 0) {
        atomicAdd(g + b, (unsigned long long) v);
        sum += v;
      }
    }
  }
  if (!WT) {
    __syncwarp();
    for (int o = 16; o > 0; o >>= 1)
      sum += __shfl_xor_sync(FULLMASK, sum, o);
    if ((threadIdx.x & 31) == 0) S->cnt[1] += sum;
    __syncwarp();
  }
}

/* Add the lanes' n to a counter of the warp's (their sum may exceed 32 bits). */
__device__ __forceinline__ void warp_count(unsigned long long *cnt, uint32_t n) {
  const uint32_t lo = __reduce_add_sync(FULLMASK, n & 0xffffu),
                 hi = __reduce_add_sync(FULLMASK, n >> 16);
  if ((threadIdx.x & 31) == 0) *cnt += ((unsigned long long) hi << 16) + lo;
}

/* The catalogue a CTA of a batched launch is working on (shared memory). */
struct TileMock {
  int nc[3];
  uint32_t base;
  float cwf[3], cwl[3];  /* cell widths: float + float residual */
};

/* Items a CTA of a batch takes at once: a share of those left, so that the
 * runs shrink towards the end and the histogram changes hands rarely.  Run i of
 * G CTAs: runs come G at a time, each 1 / (3 G) of the items left, at last of
 * TILE_RUN_MIN.  A CTA draws its run's number with one addition.  (Taking its
 * share by compare-and-swap, the CTAs of a launch wait for each other's at the
 * start: 200 mocks of 500 points 0.53 -> 0.10 ms in the kernel.  48 mocks, and
 * 256, a pass: 6.65 and 334.2 ms by compare-and-swap; 1 / (2 G) and 16 items
 * 6.49 and 336.1, 1 / (2 G) and 8 6.42 and 335.3, 1 / (3 G) and 16 6.56 and
 * 334.7, 1 / (3 G) and 8 6.49 and 334.1, 1 / (4 G) and 16 6.62 and 334.7.) */
#define TILE_RUN_MIN 8u
__device__ __forceinline__ void tile_run(uint32_t i, uint32_t G,
    uint32_t nitem, uint32_t &s0, uint32_t &s1) {
  uint32_t r = 0, sz;
  for (;;) {
    sz = (nitem - r) / (3u * G);
    if (sz <= TILE_RUN_MIN) {
      sz = TILE_RUN_MIN;
      break;
    }
    if (i < G) break;
    i -= G;
    r += G * sz;
  }
  s0 = i < (nitem - r + sz - 1u) / sz ? r + i * sz : nitem;
  s1 = nitem - s0 < sz ? nitem : s0 + sz;
}
#define TILE_CTAS 4

/* The block of an item, and the first item of a block. */
__device__ __forceinline__ uint32_t tile_block(const fcfcg_launch &L,
    uint32_t nwhole, uint32_t item) {
  return item < nwhole ? item : nwhole + ((item - nwhole) >> L.pshift);
}
__device__ __forceinline__ uint32_t tile_item(const fcfcg_launch &L,
    uint32_t nwhole, uint32_t block) {
  return block < nwhole ? block : nwhole + ((block - nwhole) << L.pshift);
}

template <int GEOM, int BIN, int WT, int BATCH, int ADJ = 0>
__global__ void __launch_bounds__(CT32_THREADS, ADJ ? 3 : TILE_CTAS)
k_tile32(const __grid_constant__ fcfcg_launch L) {
  constexpr bool SURVEY = GEOM == FCFCG_GEOM_SURVEY;
  constexpr bool F64 = BIN == BIN_F64;
  constexpr int KIND = F64 ? 3 : WT + ADJ;
  const bool cyl = !SURVEY && (F64 ? L.bintype == FCFCG_BIN_SPI : IS_SPI(BIN));
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ TileMock sh_mock;
  __shared__ uint32_t sh_run[3];     /* batch: next item, end, catalogue */
  /* edge tables: the cells in use, then the entry for all below them */
  float2 *te = (float2 *) smem;
  const EdgeTab ES = {te, L.se_lg, L.se_off, (uint32_t) L.nse - 1u},
                EP = {te + L.nse, L.pe_lg, L.pe_off, (uint32_t) L.npe - 1u};
  size_t o = ((size_t) (L.nse + L.npe) * 8 + 15) & ~(size_t) 15;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  TileWarpW *S = (TileWarpW *) (smem + o + (size_t) warp * tile_warp_bytes(KIND));
  o += (size_t) (CT32_THREADS / 32) * tile_warp_bytes(KIND);
  uint32_t *h = (uint32_t *) (smem + o);
  const uint32_t hb = (uint32_t) __cvta_generic_to_shared(h);
  /* bias of the bins' byte addresses formed from a rounded value's bits */
  LinConst C = lin_const(L);
  C.hm = 4u;
  if (HREP(WT, ADJ, BIN)) {
    C.hm = pin(4u << L.hlog);
    C.ha = hb - C.hm * TMAGIC_BITS + 4u * ((uint32_t) lane & ((1u << L.hlog) - 1u));
  } else {
    C.ha = hb - 4u * TMAGIC_BITS;
  }
  /* the lane's word behind the bins for the pairs that are not binned */
  C.spare = pin(hb + 4u * (uint32_t) ((ADJ || L.hist_smem ? L.hwords : 0) + lane));
  C.ha = pin(C.ha);
  C.slim = pin(C.slim);
  if (F64) {
    /* no tables */
  } else if (LINS(BIN)) {
    /* without a shared histogram every pair goes to tile_rest */
    C.hs = pin(ADJ || L.hist_smem ? L.tl_h : -1.f);
    C.inv = pin(C.inv);
    C.s0 = pin(C.s0);
  } else {
    C.ea = pin(C.ea);
    C.eb = pin(ADJ || L.hist_smem ? C.eb : __int_as_float(0x7f800000));
    for (int i = threadIdx.x; i < L.nse; i += blockDim.x)
      te[i] = __ldg((const float2 *) L.se + (i < L.nse - 1 ? L.se_skip + i : L.se_last));
  }
  if (IS_SMU(BIN)) {
    C.q0 = pin(C.q0);
    C.nmu = pin(C.nmu);
    C.q1 = pin(C.q1);
    C.qc = pin(C.qc);
  }
  if (IS_SPI(BIN) && !LINP(BIN))
    for (int i = threadIdx.x; i < L.npe; i += blockDim.x)
      te[L.nse + i] = __ldg((const float2 *) L.pe + (i < L.npe - 1 ? L.pe_skip + i : L.pe_last));
  if (ADJ && F64) {
    ((TileWarp64 *) S)->ga[lane] = 0;
  } else if (ADJ) {
    /* the scaled cotangent of the shared bins takes the histogram's place */
    if (L.hist_smem)
      for (int i = threadIdx.x; i < L.hlen + 32; i += blockDim.x)
        ((int2 *) h)[i] = __ldg((const int2 *) L.gtab + i);
    for (int i = 0; i < 8; i++) ((TileWarpA *) S)->ga[i][lane] = 0;
  } else if (L.hist_smem) {
    for (int i = threadIdx.x; i < (L.hwords + 32) * (WT ? 2 : 1); i += blockDim.x)
      h[i] = 0;
  }
  /* items: the blocks up to nwhole, then the rest in parts */
  const uint32_t nblk = __ldg(L.nblk_dev);
  const uint32_t nwhole = nblk > L.nsplit ? nblk - L.nsplit : 0u;
  const uint32_t nitem = tile_item(L, nwhole, nblk);
  if (blockIdx.x == 0 && threadIdx.x == 0) L.stats[4] = nblk;
  /* a warp's share of the pairs a 32-bit bin holds, less what it can add
   * between two looks at it */
  const unsigned long long share = L.hs_limit / (CT32_THREADS / 32);
  const unsigned long long lim = share > 65536u ? share - 65536u : 0u;
  if (lane < 4) S->t.cnt[lane] = 0;
  if (lane == 0) S->t.nrest = 0;
  unsigned long long added = 0;
  uint32_t cur = ~0u;
  int nq = 0;              /* all-FP64: pairs collected */
  __syncthreads();

  for (;;) {
    uint32_t item = 0;
    if (BATCH) {
      /* the CTA's run of items of one catalogue; when it is used up the
       * warps meet, and a change of catalogue hands the histogram over */
      if (lane == 0) item = atomicAdd(&sh_run[0], cur == ~0u ? 0u : 1u);
      item = __shfl_sync(FULLMASK, item, 0);
      if (cur == ~0u || item >= sh_run[1]) {
        __syncthreads();
        if (threadIdx.x == 0) {
          const uint32_t end = sh_run[2];
          uint32_t s0 = sh_run[1], s1 = s0;
          if (cur == ~0u || s0 >= end) {
            tile_run(atomicAdd(L.item_head, 1u), gridDim.x, nitem, s0, s1);
            if (s0 >= nitem) s0 = s1 = ~0u;
            sh_run[2] = s1;
          } else {
            s1 = end;
          }
          if (s0 != ~0u) {
            /* cut at the end of the first item's catalogue */
            const uint32_t mk = ((const uint2 *) L.A.bcell)[tile_block(L, nwhole, s0)].y;
            const uint32_t e = tile_item(L, nwhole,
                __ldg(L.A.bstart + __ldg(L.mbase + mk + 1)));
            if (e < s1) s1 = e;
          }
          sh_run[0] = s0;
          sh_run[1] = s1;
        }
        __syncthreads();
        const uint32_t s0 = sh_run[0];
        const uint32_t mk = s0 == ~0u ? ~0u
            : ((const uint2 *) L.A.bcell)[tile_block(L, nwhole, s0)].y;
        if (mk != cur && cur != ~0u && L.hist_smem)
          tile_handover<WT, F64>(L, h, cur, threadIdx.x, CT32_THREADS, &S->t);
        if (s0 == ~0u) break;
        if (mk != cur) {
          if (threadIdx.x < 3) {
            const fcfcg_mock *M = L.mocks + mk;
            const int k = threadIdx.x;
            sh_mock.nc[k] = M->ncell[k];
            const float f = (float) M->cw[k];
            sh_mock.cwf[k] = f;
            sh_mock.cwl[k] = (float) (M->cw[k] - (double) f);
            if (k == 0) sh_mock.base = M->cell_base;
          }
          added = 0;
        }
        __syncthreads();
        cur = mk;
        continue;
      }
    } else {
      if (lane == 0) item = atomicAdd(L.item_head, 1u);
      item = __shfl_sync(FULLMASK, item, 0);
      if (item >= nitem) break;
    }
    /* this item's share of the block's tiles: each npb-th group of 32 blocks
     * B and, in that, each npt-th tile */
    const uint32_t ab = tile_block(L, nwhole, item);
    uint32_t npt = 1, npb = 1, pt = 0, pb = 0;
    if (item >= nwhole) {
      npt = 1u << L.tshift;
      npb = 1u << (L.pshift - L.tshift);
      pt = (item - nwhole) & (npt - 1u);
      pb = ((item - nwhole) >> L.tshift) & (npb - 1u);
    }
    const uint2 ci = __ldg((const uint2 *) L.A.bcell + ab);
    const float4 *Ab = (const float4 *) L.A.blk + 2 * (size_t) ab;
    Tile T;
    T.first = __float_as_uint(__ldg(&Ab[0].w));
    T.m = (int) __float_as_uint(__ldg(&Ab[1].w));
    T.mock = ci.y;
    if (T.m == 0) continue;        /* a place left unused */
    float c2x = 0.f, c2y = 0.f, c2z = 0.f;
    if (SURVEY) {
      /* twice A's cell centre: the FP64 centre the local coordinates are
       * relative to, rounded once */
      const int cx = (int) (ci.x % (uint32_t) L.ncell[0]);
      const int cy = (int) ((ci.x / (uint32_t) L.ncell[0]) % (uint32_t) L.ncell[1]);
      const int cz = (int) (ci.x / ((uint32_t) L.ncell[0] * (uint32_t) L.ncell[1]));
      c2x = (float) (2.0 * (L.lo[0] + ((double) cx + 0.5) * L.cw[0]));
      c2y = (float) (2.0 * (L.lo[1] + ((double) cy + 0.5) * L.cw[1]));
      c2z = (float) (2.0 * (L.lo[2] + ((double) cz + 0.5) * L.cw[2]));
    }
    __syncwarp();
    {
      /* places past the block's points: a point no test passes (its squared
       * separation overflows) */
      float4 v = make_float4(-1e30f, -1e30f, -1e30f, 0.f);
      if (lane < T.m) v = __ldg((const float4 *) L.A.l4 + T.first + lane);
      float *p = (float *) S->t.p[lane >> 2] + (lane & 3);
      p[0] = v.x;
      p[4] = v.y;
      p[8] = v.z;
      group_box(S->t, v, lane, T.m);
      if (WT && !F64) {
        int2 w = make_int2(0, 0);
        if (lane < T.m) w = __ldg((const int2 *) L.A.wq + T.first + lane);
        S->aw[lane] = make_float4(__int_as_float(w.x), __int_as_float(w.y) *
                                  (ADJ ? 0x1p-30f : 1.f), v.w, 0.f);
      }
    }
    __syncwarp();
    uint32_t seq = 0, seqt = 0;
    int ntile = 0;
    /* this lane's pairs tested and in range, added up at the end of the item (at
     * each group of blocks: (s, mu) weighted +0.4 %, survey +0.9 %; at most 1024
     * per group, and 2^22 groups hold all points that there can be) */
    uint32_t cand = 0, n_in = 0;
    for (int t0 = 0; t0 < L.nsten; t0 += 32) {
      /* 32 stencil entries, one per lane: the neighbour cell's blocks */
      uint32_t nb = 0, b0 = 0, ecode = 0;
      float4 D = make_float4(0.f, 0.f, 0.f, 0.f);
      if (t0 + lane < L.nsten) {
        int nc[3] = {L.ncell[0], L.ncell[1], L.ncell[2]};
        uint32_t cbase = 0;
        if (BATCH) {
          nc[0] = sh_mock.nc[0];
          nc[1] = sh_mock.nc[1];
          nc[2] = sh_mock.nc[2];
          cbase = sh_mock.base;
        }
        const uint32_t lc = ci.x - cbase;
        const int4 so = __ldg((const int4 *) L.sten + t0 + lane);
        int q[3] = {(int) (lc % (uint32_t) nc[0]) + so.x,
                    (int) ((lc / (uint32_t) nc[0]) % (uint32_t) nc[1]) + so.y,
                    (int) (lc / ((uint32_t) nc[0] * (uint32_t) nc[1])) + so.z};
        bool in = true;
#pragma unroll
        for (int k = 0; k < 3; k++) {
          int w = 1;
          if (SURVEY) {
            in &= (q[k] >= 0) & (q[k] < nc[k]);
          } else {
            while (q[k] < 0) { q[k] += nc[k]; w--; }
            while (q[k] >= nc[k]) { q[k] -= nc[k]; w++; }
            ecode |= (uint32_t) w << (2 * k);
          }
        }
        if (in) {
          const uint32_t cb = cbase +
              ((uint32_t) q[2] * nc[1] + q[1]) * nc[0] + q[0];
          b0 = __ldg(L.B.bstart + cb);
          nb = __ldg(L.B.bstart + cb + 1) - b0;
          if (L.isauto && t0 + lane == L.tzero) {
            /* A's own cell: its block and those after it */
            nb -= ab - b0;
            b0 = ab;
          }
        }
        if (BATCH) {
          /* -offset * cell width, rounded once: the width is held as a
           * float plus its float residual */
          D.x = __fmaf_rn((float) -so.x, sh_mock.cwf[0], __fmul_rn((float) -so.x, sh_mock.cwl[0]));
          D.y = __fmaf_rn((float) -so.y, sh_mock.cwf[1], __fmul_rn((float) -so.y, sh_mock.cwl[1]));
          D.z = __fmaf_rn((float) -so.z, sh_mock.cwf[2], __fmul_rn((float) -so.z, sh_mock.cwl[2]));
        } else {
          D = __ldg((const float4 *) L.stenD + t0 + lane);
        }
        D.w = __uint_as_float(ecode);
      }
      /* entries that hold blocks and whose cell can hold a pair */
      bool visit = nb > 0;
      if (visit) {
        const float4 ac = __ldg(Ab), ah = __ldg(Ab + 1);
        const float hx = 0.5001f * (BATCH ? sh_mock.cwf[0] : L.cwf[0]),
                    hy = 0.5001f * (BATCH ? sh_mock.cwf[1] : L.cwf[1]),
                    hz = 0.5001f * (BATCH ? sh_mock.cwf[2] : L.cwf[2]);
        const float gx = fmaxf(fabsf(ac.x + D.x) - (ah.x + hx) - L.box_eps, 0.f),
                    gy = fmaxf(fabsf(ac.y + D.y) - (ah.y + hy) - L.box_eps, 0.f),
                    gz = fmaxf(fabsf(ac.z + D.z) - (ah.z + hz) - L.box_eps, 0.f);
        if (cyl)
          visit = (gz < L.p_lim) & (fmaf(gy, gy, gx * gx) < L.s_lim);
        else
          visit = fmaf(gz, gz, fmaf(gy, gy, gx * gx)) < L.s_lim;
      }
      uint32_t cells = __ballot_sync(FULLMASK, visit);
      __syncwarp();
      S->t.sd[lane] = D;
      S->t.si[lane] = make_uint2(b0, nb);
      __syncwarp();
      while (cells) {
       const int e = __ffs(cells) - 1;
       cells &= cells - 1u;
       const float4 d = S->t.sd[e];
       const uint2 eb = S->t.si[e];
       const bool own = L.isauto && t0 + e == L.tzero;
       T.code = __float_as_uint(d.w);
       for (uint32_t g = 0; g < eb.y; g += 32) {
        if ((seq++ & (npb - 1u)) != pb) continue;
        /* 32 blocks, one per lane: can a pair with A's block count? */
        bool near = false;
        uint32_t bfirst = 0, groups = 0;
        int bcnt = 0;
        if (g + lane < eb.y) {
          const float4 ac = __ldg(Ab), ah = __ldg(Ab + 1);
          const float4 *Bb = (const float4 *) L.B.blk +
              2 * (size_t) (eb.x + g + lane);
          const float4 bc = __ldg(Bb), bh = __ldg(Bb + 1);
          bfirst = __float_as_uint(bc.w);
          bcnt = (int) __float_as_uint(bh.w);
          /* the boxes' distance, less a slack above its rounding and the
           * pair arithmetic's: no pair of the blocks is closer */
          const float gx = fmaxf(fabsf(ac.x - (bc.x - d.x)) - (ah.x + bh.x) - L.box_eps, 0.f),
                      gy = fmaxf(fabsf(ac.y - (bc.y - d.y)) - (ah.y + bh.y) - L.box_eps, 0.f),
                      gz = fmaxf(fabsf(ac.z - (bc.z - d.z)) - (ah.z + bh.z) - L.box_eps, 0.f);
          if (cyl)
            near = (gz < L.p_lim) & (fmaf(gy, gy, gx * gx) < L.s_lim);
          else
            near = fmaf(gz, gz, fmaf(gy, gy, gx * gx)) < L.s_lim;
          if (LOSCUT(GEOM, BIN) && near)
            near = !los_apart(L, c2x, c2y, c2z, ac, ah, bc.x - d.x,
                              bc.y - d.y, bc.z - d.z, bh);
          if (near && npt > 1 && !F64) {
            groups = (1u << ((T.m + 3) >> 2)) - 1u;
          } else if (near) {
            /* which groups of four of A's points can */
            const float bx = bc.x - d.x, by = bc.y - d.y, bz = bc.z - d.z;
            const float hx = bh.x + L.box_eps, hy = bh.y + L.box_eps,
                        hz = bh.z + L.box_eps;
#pragma unroll 2
            for (int q = 0; q < 8; q++) {
              const float4 c = S->t.gc[q], r = S->t.gh[q];
              const float gx = fmaxf(fabsf(c.x - bx) - (r.x + hx), 0.f),
                          gy = fmaxf(fabsf(c.y - by) - (r.y + hy), 0.f),
                          gz = fmaxf(fabsf(c.z - bz) - (r.z + hz), 0.f);
              bool in;
              if (cyl)
                in = (gz < L.p_lim) & (fmaf(gy, gy, gx * gx) < L.s_lim);
              else
                in = fmaf(gz, gz, fmaf(gy, gy, gx * gx)) < L.s_lim;
              if (LOSCUT(GEOM, BIN) && in)
                in = !los_apart(L, c2x, c2y, c2z, c, r, bx, by, bz, bh);
              if (in) groups |= 1u << q;
            }
            near = groups != 0u;
          }
        }
        uint32_t todo = __ballot_sync(FULLMASK, near);
        if (npt > 1) {
          /* by single tiles: this part's */
          near &= ((seqt + (uint32_t) __popc(todo & ((1u << lane) - 1u))) &
                   (npt - 1u)) == pt;
          seqt += (uint32_t) __popc(todo);
          todo = __ballot_sync(FULLMASK, near);
        }
        if (ADJ && !F64) ntile += __popc(todo);
        added += 1024u * (uint32_t) __popc(todo);
        /* the pairs tested, of this lane's block: the fours taken, the last one
         * of fewer points perhaps */
        if (near) {
          const int na = 4 * __popc(groups);
          cand += (uint32_t) ((groups >> ((T.m - 1) >> 2) ? na - (-T.m & 3) : na) * bcnt);
        }
        while (todo) {
          const int j = __ffs(todo) - 1;
          todo &= todo - 1u;
          const uint32_t f = __shfl_sync(FULLMASK, bfirst, j);
          const int n = __shfl_sync(FULLMASK, bcnt, j);
          T.gm = __shfl_sync(FULLMASK, groups, j);
          const bool self = own && g + (uint32_t) j == 0;
          /* lanes past the block: a point no test passes */
          T.bx = T.by = T.bz = 1e30f;
          T.bj = f + (uint32_t) lane;
          T.wi = 0;
          T.wr = T.wf = 0.f;
          if (lane < n) {
            const float4 v = __ldg((const float4 *) L.B.l4 + T.bj);
            T.bx = v.x - d.x;
            T.by = v.y - d.y;
            T.bz = v.z - d.z;
            if (WT && !F64) {
              const int2 w = __ldg((const int2 *) L.B.wq + T.bj);
              T.wi = w.x;
              T.wr = __int_as_float(w.y) * (ADJ ? 0x1p-30f : 1.f);
              T.wf = v.w;
            }
          }
          T.ilim = self ? lane : 32;
          if (F64) T.ilim = lane < n ? min(T.ilim, T.m) : 0;
          bool sp = self;
          if (SURVEY && !F64) {
            T.vx = fmaf(2.f, T.bx, c2x);
            T.vy = fmaf(2.f, T.by, c2y);
            T.vz = fmaf(2.f, T.bz, c2z);
            const float r2 = 0.25f * fmaf(T.vz, T.vz, fmaf(T.vy, T.vy, T.vx * T.vx));
            if (!IS_ISO(BIN))
              sp |= __any_sync(FULLMASK, r2 < L.near2) != 0;
            if (LOSCUT(GEOM, BIN)) {
              T.ux = T.uy = T.uz = T.lh = 0.f;
              T.lP = FLT_MAX;          /* near the observer: no cut */
              if (r2 > L.los_r2min && lane < n) {
                const float ir = rsq_ftz(r2);
                T.ux = 0.5f * T.vx * ir;
                T.uy = 0.5f * T.vy * ir;
                T.uz = 0.5f * T.vz * ir;
                T.lh = L.los_h * ir;
                T.lP = fmaf(L.los_pr, ir, L.los_p);
              }
            }
          }
          if constexpr (F64) {
            tile_pairs64<GEOM, WT, ADJ>(L, T, (TileWarp64 *) S, h, nq, n_in);
          } else {
            uint32_t rest;
            long long gb = 0;     /* adjoint: this lane's point's terms */
            if (sp)
              rest = tile_pairs<GEOM, BIN, WT, ADJ, true>(L, C, T, S, hb, ES,
                                                          EP, n_in, gb);
            else
              rest = tile_pairs<GEOM, BIN, WT, ADJ, false>(L, C, T, S, hb, ES,
                                                           EP, n_in, gb);
            if (ADJ && gb) atomicAdd(L.dB + T.bj, (double) gb * L.gunitB);
            if (__any_sync(FULLMASK, rest != 0u)) {
              if (!ADJ && !L.hist_smem)
                rest = tile_global<GEOM, BIN, WT>(L, T, S, rest, ES, EP);
              /* (in place where the loop has many values to keep: the call
               * saves them, 0.9 % of a weighted (s, mu) count; the others gain
               * 2 % by the registers, survey (s_perp, pi) 1.6 %) */
              const uint32_t code = T.code | T.mock << 6;
              if (WT && !IS_SPI(BIN))
                tile_rest<WT, ADJ>(L, &S->t, rest, T.first, T.bj, code);
              else
                tile_rest_call<WT, ADJ>(L, &S->t, rest, T.first, T.bj, code);
            }
          }
        }
        if (ADJ && !F64) {
          /* a term is at most 2^52 (2^52 itself for a weight and an entry of
           * 1), a tile adds 32 of them to a point's eight words, which
           * adj_flush adds up four at a time in 64 bits: out after at most 95 +
           * 32 tiles, 127 x 16 x 2^52 < 2^63 */
          if (ntile > 127 - 32) {
            adj_flush(L, (TileWarpA *) S, T.first, T.m);
            ntile = 0;
          }
        }
        if (!WT && !ADJ && added > lim && L.hist_smem) {
          /* a warp that may have added its share of what a 32-bit bin holds
           * hands the CTA's bins over */
          tile_handover<WT>(L, h, T.mock, lane, 32, &S->t);
          added = 0;
        }
       }
      }
    }
    warp_count(&S->t.cnt[0], cand);
    if (WT || (F64 && !L.hist_smem)) warp_count(&S->t.cnt[1], n_in);
    if (ADJ && F64) {
      double &ga = ((TileWarp64 *) S)->ga[lane];
      __syncwarp();
      if (lane < T.m && ga != 0.0) atomicAdd(L.dA + T.first + lane, ga);
      ga = 0;
      __syncwarp();
    } else if (ADJ) {
      adj_flush(L, (TileWarpA *) S, T.first, T.m);
    }
  }
  if (F64 && !ADJ) {
    uint32_t n_in = 0;
    __syncwarp();
    bin64<WT>(L, (TileWarp64 *) S, h, 0, nq, n_in);
    n_in = __reduce_add_sync(FULLMASK, n_in);
    if (lane == 0) S->t.cnt[1] += n_in;
  }
  if (!BATCH && !ADJ) {
    __syncthreads();
    if (L.hist_smem)
      tile_handover<WT, F64>(L, h, 0, threadIdx.x, CT32_THREADS, &S->t);
  }
  if (!F64) rest_flush<WT, ADJ>(L, &S->t, 0u, 0u, 0u, 0u);
  __syncwarp();
  if (lane < 4) atomicAdd(L.stats + lane, S->t.cnt[lane]);
}

#endif

// Contour tracing on the ultra-fine grid, tile by tile.
//
// The level codes at a box's four corners say for every level which of its
// edges the level's contours enter and leave by, so a contour can be followed
// from box to box without any table of crossings: a CTA stages the codes of
// 128 x 64 boxes in shared memory and walks every contour piece of its tile
// there.  A crossing's number is its edge's offset (the reference's edge order;
// the offsets of 16-edge chunks come from a count and a scan, those inside a
// chunk from the codes) plus its level's place on the edge, known to every CTA
// that meets the edge, so pieces of neighbouring tiles link by number.  What
// leaves the tile kernel is each crossing's (chain, place) and position and
// one record per chain; lists are ranked over the chains only.
//
// This took the place of emitting every (edge, level), sorting by level, a
// (level, box) hash for the successors and a walk over the successors in
// global memory with splitters at every 16th crossing.  Crossings are numbered
// in edge order instead of level by level: within a level that is the same
// order, and only contours (a few thousand) are sorted by level at the end.
//
// Measured (B200), contours plus residual at 1024^2, 25M crossings: the part
// from the counts to the walk layout took 6.7 ms and takes 3.3 ms (k_cr_count
// 0.24, k_tr_walk 1.35, ranking 0.41, k_tr_place 1.09), the whole recontouring
// 13.3 and 9.5 ms (8.5 with later changes to the renode passes and the field);
// beta-plane from a field at 256^2 3.2 and 1.8 ms (1.50).
// k_tr_walk is bound by the latency of its walks (16k of a tile's 31k cycles:
// 23 chains of 32 crossings, some 190 cycles a step, in one warp; the rest is
// staging and the offsets), k_tr_place by issue (63 % of the slots).
#pragma once

#include "common.cuh"
#include "state.cuh"

namespace casl {

// The grid whose edges are numbered: nxu columns, periodic in x; rows
// 0..nrow-1, periodic (congen.f90) or open in y (the extended grid of
// econgen.f90).  x-line edges (ix, r)-(ix, r+1), r < ner, are numbered column
// by column, then y-line edges (ix, r)-(ix+1, r) row by row, rows ylo ..
// ylo+nyl-1, as congen.f90:200-254 and econgen.f90:238-348 do.  Chunks: 16
// consecutive edges of one column (nseg per column), then of one row.
struct CrGrid {
  int nxu, nrow, ner, nseg, ylo, nyl;
  int nbr;               // rows of boxes
  int periodic;
  int cmin, cmax;        // codes are clamped to levbeg-1 .. levend
  long long ld;          // codes per column (a multiple of 256)
  long long ncx;         // x-line chunks
  const unsigned short *lc;
};
inline long long cr_chunks(const CrGrid &g) { return g.ncx + (long long)g.nyl * (g.nxu / 16); }

// |a - b| of two pairs of unsigned 16-bit values: the halves' maxima less their
// minima, which cannot borrow.  __vabsdiffu2 is several times the instructions
// (k_cr_count at 1024^2 314 us with it, 241 so).
__device__ __forceinline__ unsigned absdiff2(unsigned a, unsigned b) {
  return __vmaxu2(a, b) - __vminu2(a, b);
}

// Crossings per chunk.  A thread takes 8 rows of 17 columns as 16-byte loads
// (lanes along the rows: coalesced) and counts with packed 16-bit differences:
// both kinds of chunk from one read of the codes.  8 warps cover 128 columns,
// so that the y-line counts of a row are written as whole sectors.  *wide (zero on
// entry) is set when a chunk has more than 16-bit places can number.
constexpr int TR_NARROW = 65534;
__global__ void __launch_bounds__(256, 2) k_cr_count(CrGrid g, int *__restrict__ cnt,
                                                     int *__restrict__ wide) {
  CASL_PDL_ENTRY();
  __shared__ int Y[256][9];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int nbx = g.nxu / 128;
  const int bx = blockIdx.x % nbx, by = blockIdx.x / nbx;
  const int r0 = by * 256 + 8 * lane, ix0 = bx * 128 + w * 16;
  const unsigned lo2 = (unsigned)g.cmin * 0x10001u, hi2 = (unsigned)g.cmax * 0x10001u;
  const int nv = min(max(g.ner - r0, 0), 8);  // x-line edges in range
  int rn = r0 + 8;                            // the row after
  if (rn >= g.nrow) rn = g.periodic ? rn - g.nrow : g.nrow - 1;
  int acc[8];
#pragma unroll
  for (int k = 0; k < 8; k++) acc[k] = 0;
  unsigned p[4] = {0, 0, 0, 0};
#pragma unroll
  for (int i = 0; i <= 16; i++) {
    int ix = ix0 + i;
    if (ix >= g.nxu) ix -= g.nxu;
    const unsigned short *col = g.lc + (long long)ix * g.ld;
    const uint4 v = __ldg(reinterpret_cast<const uint4 *>(col + r0));
    unsigned c[5] = {v.x, v.y, v.z, v.w, 0};
#pragma unroll
    for (int k = 0; k < 4; k++) c[k] = __vminu2(__vmaxu2(c[k], lo2), hi2);
    if (i < 16) {
      c[4] = __shfl_down_sync(0xffffffffu, c[0], 1);
      if (lane == 31 || nv < 8 || rn != r0 + 8)
        c[4] = (unsigned)min(max((int)__ldg(col + rn), g.cmin), g.cmax);
      int s = 0;
#pragma unroll
      for (int k = 0; k < 4; k++) {
        const unsigned d = absdiff2(c[k], __funnelshift_r(c[k], c[k + 1], 16));
        s += (2 * k < nv ? d & 0xffffu : 0u) + (2 * k + 1 < nv ? d >> 16 : 0u);
      }
      s += __shfl_down_sync(0xffffffffu, s, 1);
      const int seg = r0 >> 4;
      if (!(lane & 1) && seg < g.nseg) {
        cnt[(long long)ix * g.nseg + seg] = s;
        if (s > TR_NARROW) *wide = 1;
      }
    }
    if (i > 0) {
#pragma unroll
      for (int k = 0; k < 4; k++) {
        const unsigned d = absdiff2(p[k], c[k]);
        acc[2 * k] += d & 0xffffu;
        acc[2 * k + 1] += d >> 16;
      }
    }
#pragma unroll
    for (int k = 0; k < 4; k++) p[k] = c[k];
  }
#pragma unroll
  for (int k = 0; k < 8; k++) Y[8 * lane + k][w] = acc[k];
  __syncthreads();
  const int row = by * 256 + threadIdx.x;
  if (row >= g.ylo && row < g.ylo + g.nyl) {
    const int *y = Y[threadIdx.x];
    int4 *o = reinterpret_cast<int4 *>(cnt + g.ncx + (long long)(row - g.ylo) * (g.nxu / 16) + bx * 8);
    o[0] = make_int4(y[0], y[1], y[2], y[3]);
    o[1] = make_int4(y[4], y[5], y[6], y[7]);
    int most = 0;
#pragma unroll
    for (int k = 0; k < 8; k++) most = max(most, y[k]);
    if (most > TR_NARROW) *wide = 1;
  }
}

// ---------------------------------------------------------------------------
// Tiles
// ---------------------------------------------------------------------------
// Tiles of 128 x 64 boxes with chains cut at every 32nd line: one walking warp
// of a tile then has some 23 lanes at work.  With 64 x 64 tiles and chains
// across the whole tile (5 lanes, twice the steps) k_tr_walk took 1.9 ms, with
// 128 x 64 and uncut chains 1.8 ms.
constexpr int TX = 128, TY = 64;  // boxes of a tile
constexpr int TS = TY + 2;        // codes per staged column (33 words: no common bank)
constexpr int TCX = TY / 16, TCY = TX / 16;           // chunks per column, per row
constexpr int TQX = (TX + 1) * TCX, TQY = (TY + 1) * TCY;  // x-line and y-line chunks met
constexpr int TB = 32;             // chains end at every TB-th x-line and y-line
constexpr int TR_NT = 256;        // threads per tile
// Starts listed at once (2048 words leave room for the three CTAs an SM that 512
// leave; 128^2, 2000 levels: k_tr_walk 845, 560, 405 us with 512, 1024, 2048),
// crossings listed at once, and the crossings an edge from which edges are
// listed instead (64^2, 1000 levels: k_tr_place 420 us from 4, 575 from 8 on).
constexpr int TR_SCAP = 2048, TR_GCAP = 2048, TR_MANY = 4;
// column of staged point m (m / TS for every m < (TX + 2) * TS)
__device__ __forceinline__ int tr_col(int m) { return (m * 993) >> 16; }

// A chain: crossings that follow one another, from one on every TB-th grid
// line (or one that leaves a saddle box) to the last before the next such
// line or saddle box, or once around a contour that meets neither.
struct TrArgs {
  CrGrid g;
  const int *off;        // chunk offsets
  int2 *own;             // per crossing: chain, place in it
  int4 *chain;           // next chain's first crossing (-1: ends), length, least crossing, last crossing
  int *clev;             // per chain: level
  int *nchain, cap;      // chains, and the most of them and of eidx
  int *eidx;             // crossings entering saddle boxes ...
  long long *eslot;      // ... and the boxes' two out-crossings, lower << 32 | higher
  int *nend;
  int *err;
};

// The codes of TX x TY boxes ((TX+1) columns x (TY+1) rows) from (ix0, j0);
// whether any two differ.
__device__ __forceinline__ bool tr_stage(const CrGrid &g, int ix0, int j0, unsigned short *C) {
  int differ = 0;
  const int ref = min(max((int)__ldg(g.lc + (long long)ix0 * g.ld + j0), g.cmin), g.cmax);
  const unsigned lo2 = (unsigned)g.cmin * 0x10001u, hi2 = (unsigned)g.cmax * 0x10001u;
  constexpr int V = TY / 8;  // 16-byte vectors per column
  for (int q = threadIdx.x; q < (TX + 1) * (V + 1); q += TR_NT) {
    const bool last = q >= (TX + 1) * V;  // the row after the tile
    const int part = q & (V - 1), col = last ? q - (TX + 1) * V : q / V;
    int ix = ix0 + col;
    if (ix >= g.nxu) ix -= g.nxu;
    const unsigned short *src = g.lc + (long long)ix * g.ld;
    if (!last) {
      const uint4 v = __ldg(reinterpret_cast<const uint4 *>(src + j0 + 8 * part));
      unsigned w[4] = {v.x, v.y, v.z, v.w};
      unsigned *d = reinterpret_cast<unsigned *>(C + col * TS + 8 * part);
#pragma unroll
      for (int k = 0; k < 4; k++) {
        w[k] = __vminu2(__vmaxu2(w[k], lo2), hi2);
        d[k] = w[k];
        differ |= w[k] != (unsigned)ref * 0x10001u;
      }
    } else {
      int r = j0 + TY;
      if (r >= g.nrow) r = g.periodic ? r - g.nrow : g.nrow - 1;
      const int v = min(max((int)__ldg(src + r), g.cmin), g.cmax);
      *reinterpret_cast<unsigned *>(C + col * TS + TY) = (unsigned)v * 0x10001u;
      differ |= v != ref;
    }
  }
  return __syncthreads_or(differ) != 0;
}

// Number of the x-line chunk (column col, rows 16 sg ..) or y-line chunk (row,
// columns 16 sg ..) of the tile at (ix0, j0); -1 where the edges have none.
__device__ __forceinline__ long long tr_xchunk(const CrGrid &g, int ix0, int j0, int col, int sg) {
  int ix = ix0 + col;
  if (ix >= g.nxu) ix -= g.nxu;
  const int seg = (j0 >> 4) + sg;
  return seg < g.nseg ? (long long)ix * g.nseg + seg : -1;
}
__device__ __forceinline__ long long tr_ychunk(const CrGrid &g, int ix0, int j0, int row, int sg) {
  int r = j0 + row;
  if (g.periodic && r >= g.nrow) r -= g.nrow;
  return r >= g.ylo && r < g.ylo + g.nyl ? g.ncx + (long long)(r - g.ylo) * (g.nxu / 16) + (ix0 >> 4) + sg
                                         : -1;
}

constexpr int TR_Y = (TX + 1) * TS;  // y-lines' places follow the x-lines'
template <class Rel>
struct TrTile {
  const unsigned short *C;    // codes, [column][row], row length TS
  const Rel *rel;             // by an edge's first point: crossings of its chunk before it
  const int *cb;              // chunk offsets: x-lines [column][TCX], y-lines [row][TCY]
  int th;                     // box rows of the tile (TY but at an open top)
  bool open0, open1;          // no boxes below / above the tile (a grid open in y)
};
// A contour of level l on its way through an edge: high values lie to the left
// of its direction (congen.f90:211-252), so the edge runs from the point P on
// the left (code >= l) to Q on the right (code < l, namely lo); v is the step
// of C to the far side of the box ahead, +-TS along x, +-1 along y.
struct TrPos {
  int P, Q, v, lo;
};
template <class Rel>
__device__ __forceinline__ TrPos tr_at(const TrTile<Rel> &T, int m, int y, int l) {
  const int n = m + (y ? TS : 1);
  const bool fwd = (int)T.C[m] >= l;
  TrPos p;
  p.P = fwd ? m : n;
  p.Q = fwd ? n : m;
  p.v = y ? (fwd ? 1 : -1) : (fwd ? -TS : TS);
  p.lo = T.C[p.Q];
  return p;
}
// What p's edge is: the places in cb and rel of its crossings' numbers, and
// whether chains end at it.
struct TrEdge {
  int q, r;
  bool line, open;  // open: a first or last row that no level reaches
};
template <class Rel>
__device__ __forceinline__ TrEdge tr_edge(const TrTile<Rel> &T, const TrPos &p) {
  const int m = min(p.P, p.Q), col = tr_col(m), row = m - col * TS;
  const bool y = p.v == 1 || p.v == -1;
  TrEdge e;
  e.q = y ? TQX + row * TCY + (col >> 4) : col * TCX + (row >> 4);
  e.r = m + (y ? TR_Y : 0);
  e.line = ((y ? row : col) & (TB - 1)) == 0;
  e.open = y && ((row == 0 && T.open0) || (row == T.th && T.open1));
  return e;
}
template <class Rel>
__device__ __forceinline__ int tr_id(const TrTile<Rel> &T, const TrPos &p, int l) {
  const TrEdge e = tr_edge(T, p);
  return T.cb[e.q] + (int)T.rel[e.r] + l - p.lo - 1;
}
// Through the box ahead, whose far points have codes cl (left) and cr, to its
// exit: straight on when the left one is high and the right one low, right
// when both are high, left when both are low (selects only: the lanes of a
// walking warp turn differently).  Not at a saddle (left low, right high).
__device__ __forceinline__ void tr_step(TrPos &p, int l, int cl, int cr) {
  const int fl = p.P + p.v, fr = p.Q + p.v, u = p.P - p.Q;  // u: a quarter turn left of v
  const bool hl = cl >= l, hr = cr >= l;
  p.P = hl ? (hr ? fr : fl) : p.P;
  p.Q = hr ? p.Q : (hl ? fr : fl);
  p.lo = hr ? p.lo : (hl ? cr : cl);
  p.v = hl == hr ? (hl ? -u : u) : p.v;
}
// Follows level l from the edge (m, y) as chain c; the chain's length.
// `loop`: a contour that meets no line where chains end.  A step's four reads
// of shared memory are issued together: the crossing's number and the two
// points ahead (which lie outside the staged codes, but inside the block's
// shared memory, where the walk ends).
template <class Rel>
__device__ __forceinline__ int tr_walk(const TrArgs &a, const TrTile<Rel> &T, int m, int y, int l, int c,
                                       bool loop) {
  TrPos p = tr_at(T, m, y, l);
  int first = -1, last = -1, mn = 0x7fffffff, k = 0, nxt = -1;
  while (true) {
    const TrEdge e = tr_edge(T, p);
    const int nb = T.cb[e.q], nr = T.rel[e.r], cl = T.C[p.P + p.v], cr = T.C[p.Q + p.v];
    const int id = nb + nr + l - p.lo - 1;
    // (no level reaches an open grid's first and last rows, and no walk is
    // endless: otherwise the codes are not the counted ones)
    if (e.open || k > (1 << 20) || (loop && e.line)) {
      atomicExch(a.err, CASL_EINVAL);
      break;
    }
    if (k > 0 && (loop ? id == first : e.line)) {
      nxt = id;
      break;
    }
    if (k == 0) first = id;
    a.own[id] = make_int2(c, k++);
    mn = min(mn, id);
    last = id;
    if (cl < l && cr >= l) {
      // a saddle's exits: left of the near left point and right of the near
      // right one, the edges (P, far left) and (far right, Q)
      const int fl = p.P + p.v, fr = p.Q + p.v, u = p.P - p.Q;
      const int e0 = tr_id(T, TrPos{p.P, fl, u, cl}, l), e1 = tr_id(T, TrPos{fr, p.Q, -u, p.lo}, l);
      const int s = atomicAdd(a.nend, 1);
      if (s < a.cap) {
        a.eidx[s] = id;
        a.eslot[s] = (long long)(((unsigned long long)min(e0, e1) << 32) | (unsigned int)max(e0, e1));
      } else {
        atomicExch(a.err, CASL_ECAPACITY);
      }
      break;
    }
    tr_step(p, l, cl, cr);
  }
  a.chain[c] = make_int4(nxt, k, mn, last);
  a.clev[c] = l;
  return k;
}
// Whether level l's crossing of x-line edge m, which moves to the left, is the
// least such one of a contour that meets no line where chains end (most walks
// end after a step or two, at the next x-line to the left).
template <class Rel>
__device__ __forceinline__ bool tr_least(const TrArgs &a, const TrTile<Rel> &T, int m, int l) {
  TrPos p = tr_at(T, m, 0, l);
  int first = -1;
  for (int guard = 0; guard <= (1 << 20); guard++) {
    const TrEdge e = tr_edge(T, p);
    if (e.line || e.open) return false;
    if (p.v == -TS) {
      const int id = T.cb[e.q] + (int)T.rel[e.r] + l - p.lo - 1;
      if (guard == 0) first = id;
      else if (id == first) return true;
      else if (id < first) return false;
    }
    const int cl = T.C[p.P + p.v], cr = T.C[p.Q + p.v];
    if (cl < l && cr >= l) return false;
    tr_step(p, l, cl, cr);
  }
  atomicExch(a.err, CASL_EINVAL);
  return false;
}

// The starts of a tile's chains: the crossings of every TB-th line that enter a
// box of the tile, and the out-crossings of its saddle boxes on other lines.
// line(m, y, c0, c1, which, last): an edge of such a line, from point m (y-line
// when y) with codes c0, c1 at its ends, on line `which` of 0..last;
// range(m, y, lo, hi): levels lo+1 .. hi that leave a saddle box by edge (m, y).
template <class Rel, class Line, class Range>
__device__ __forceinline__ void tr_starts(const TrTile<Rel> &T, Line line_f, Range range) {
  const unsigned short *C = T.C;
  const int tid = threadIdx.x, th = T.th;
  auto word = [&](int p) { return *reinterpret_cast<const unsigned *>(C + p); };
  constexpr int LX = (TX / TB + 1) * TY, LY = (TY / TB + 1) * TX;
  for (int q = tid; q < LX + LY; q += TR_NT) {
    const bool y = q >= LX;
    const int line = y ? (q - LX) / TX * TB : q / TY * TB, at = y ? (q - LX) % TX : q % TY;
    const int m = y ? at * TS + line : line * TS + at;
    const bool ok = y ? line < th || (th == TY && line == TY) : at < th;
    if (!ok || (y && ((line == 0 && T.open0) || (line == th && T.open1)))) continue;
    line_f(m, (int)y, (int)C[m], (int)C[m + (y ? TS : 1)], line, y ? TY : TX);
  }
  // saddles, two rows of boxes at a time; a thread's boxes: half a column
  const int bi = tid >> 1, bj0 = (TY / 2) * (tid & 1);
  int m = bi * TS + bj0;
  unsigned a0 = word(m), b0 = word(m + TS);
  for (int j = bj0; j < bj0 + TY / 2; j += 2, m += 2) {
    const unsigned a2 = word(m + 2), b2 = word(m + TS + 2);
    const unsigned a1 = __funnelshift_r(a0, a2, 16), b1 = __funnelshift_r(b0, b2, 16);
    const unsigned sd = __vcmpgtu2(__vminu2(a0, b1), __vmaxu2(b0, a1)) |
                        __vcmpgtu2(__vminu2(b0, a1), __vmaxu2(a0, b1));
    if (sd) {
      for (int h = 0; h < 2; h++) {
        const int jj = j + h, mm = m + h;
        if (jj >= th) break;
        const int c00 = C[mm], c10 = C[mm + TS], c01 = C[mm + 1], c11 = C[mm + TS + 1];
        const int xl = max(c10, c01), xh = min(c00, c11), yl = max(c00, c11), yh = min(c10, c01);
        if (xh > xl) {  // exits left and right
          if (bi % TB) range(mm, 0, xl, xh);
          if ((bi + 1) % TB) range(mm + TS, 0, xl, xh);
        }
        if (yh > yl) {  // exits bottom and top
          if (jj % TB) range(mm, 1, yl, yh);
          if ((jj + 1) % TB && jj + 1 < th) range(mm + 1, 1, yl, yh);
        }
      }
    }
    a0 = a2;
    b0 = b2;
  }
}
// The levels of a line's edge that start there: c1 high, to the right or down;
// c0 high, to the left or up.  On the tile's own sides only those that enter it.
template <class Range>
__device__ __forceinline__ void tr_line_starts(int m, int y, int c0, int c1, int line, int last,
                                               Range range) {
  if ((y ? line > 0 : line < last) && c1 > c0) range(m, y, c0, c1);
  if ((y ? line < last : line > 0) && c0 > c1) range(m, y, c1, c0);
}

template <class Rel>
struct TrSmem {
  unsigned short before[TS + 6];  // a step down or to the left of the tile reads here
  unsigned short C[TR_Y];
  alignas(4) Rel rel[2 * TR_Y];
  int cb[TQX + TQY];
  unsigned int slist[TR_SCAP];
};
// A tile is one CTA's (blockIdx.x), or several's when its crossings are many and
// tiles few (blockIdx.y, tr_slices): each then stages the tile and takes its
// share of the starts.
// Rel: places inside a chunk in 16 bits, or in 32 where some chunk has more
// crossings: 98 KB of shared memory for 64, 2 CTAs an SM for 3 (25M crossings at
// 1024^2: 2.12 ms with 32 bits, 1.35 with 16).
template <class Rel>
__global__ void __launch_bounds__(TR_NT, sizeof(Rel) == 2 ? 3 : 2) k_tr_walk(TrArgs a) {
  CASL_PDL_ENTRY();
  extern __shared__ __align__(16) unsigned char tr_smem[];
  TrSmem<Rel> &sm = *reinterpret_cast<TrSmem<Rel> *>(tr_smem);
  unsigned short *C = sm.C;
  Rel *rel = sm.rel;
  int *cb = sm.cb;
  unsigned int *slist = sm.slist;
  __shared__ int nstart, nvis, nnode, base, total;
  const CrGrid &g = a.g;
  const int tid = threadIdx.x;
  const int ntx = g.nxu / TX;
  const int ix0 = (int)(blockIdx.x % ntx) * TX, j0 = (int)(blockIdx.x / ntx) * TY;
  if (tid == 0) nstart = nvis = nnode = 0;
  for (int q = tid; q < TQX + TQY; q += TR_NT) {
    const long long ch = q < TQX ? tr_xchunk(g, ix0, j0, q / TCX, q % TCX)
                                 : tr_ychunk(g, ix0, j0, (q - TQX) / TCY, (q - TQX) % TCY);
    cb[q] = ch >= 0 ? __ldg(a.off + ch) : 0;
  }
  if (!tr_stage(g, ix0, j0, C)) return;
  const int th = min(TY, g.nbr - j0);
  const TrTile<Rel> T{C, rel, cb, th, !g.periodic && j0 == 0, !g.periodic && j0 + th == g.nbr};
  // Places inside the chunks: prefix sums of the codes' differences, two rows
  // at a time (16-bit halves), and the crossings of the edges between two of
  // the tile's boxes, all of which enter one of them.  (Rows of a grid open in y
  // past its last have codes of any kind, and sums that nothing reads.)
  auto word = [&](int p) { return *reinterpret_cast<const unsigned *>(C + p); };
  constexpr bool WIDE = sizeof(Rel) == 4;
  int nodes = 0;
  for (int q = tid; q < TQX; q += TR_NT) {
    const int col = q / TCX, r0 = 16 * (q % TCX), p0 = col * TS + r0;
    const bool inner = col > 0 && col < TX;
    unsigned w = word(p0), run = 0;
#pragma unroll
    for (int k = 0; k < 8; k++) {
      const unsigned n = word(p0 + 2 * k + 2), d = absdiff2(w, __funnelshift_r(w, n, 16));
      const unsigned d0 = d & 0xffffu, d1 = d >> 16;
      if constexpr (WIDE) {
        rel[p0 + 2 * k] = run;
        rel[p0 + 2 * k + 1] = run + d0;
      } else {
        *reinterpret_cast<unsigned *>(rel + p0 + 2 * k) = (run & 0xffffu) | (run + d0) << 16;
      }
      if (inner) nodes += (r0 + 2 * k < th ? d0 : 0u) + (r0 + 2 * k + 1 < th ? d1 : 0u);
      run += d0 + d1;
      w = n;
    }
  }
  for (int q = tid; q < (TY / 2 + 1) * TCY; q += TR_NT) {
    const int r = 2 * (q / TCY), p0 = 16 * (q % TCY) * TS + r;
    unsigned w = word(p0), lo = 0, hi = 0;  // (16 bits: both rows' sums in lo)
#pragma unroll
    for (int k = 0; k < 16; k++) {
      const unsigned n = word(p0 + (k + 1) * TS), d = absdiff2(w, n);
      if constexpr (WIDE) {
        rel[TR_Y + p0 + k * TS] = lo;
        rel[TR_Y + p0 + k * TS + 1] = hi;
        lo += d & 0xffffu;
        hi += d >> 16;
      } else {
        *reinterpret_cast<unsigned *>(rel + TR_Y + p0 + k * TS) = lo;
        lo = __vadd2(lo, d);
      }
      w = n;
    }
    if (r > 0 && r < th) nodes += WIDE ? lo : lo & 0xffffu;
    if (r + 1 < th) nodes += WIDE ? hi : lo >> 16;
  }
  __syncthreads();
  auto entry = [&](int m, int y, int l) { return (unsigned)(m << 1 | y) << 16 | (unsigned)l; };
  // the walks of the list's first ns starts (consecutive lanes: a walking
  // warp's cost is that of its longest walk)
  int mine = 0;
  auto walk_list = [&](int ns) {
    if (tid == 0) base = ns ? atomicAdd(a.nchain, ns) : 0;
    __syncthreads();
    for (int s = tid; s < ns; s += TR_NT) {
      const int c = base + s;
      const unsigned w = slist[s];
      if (c < a.cap) mine += tr_walk(a, T, (int)(w >> 17), (int)(w >> 16) & 1, (int)(w & 0xffffu), c, false);
      else atomicExch(a.err, CASL_ECAPACITY);
    }
  };
  // What does not fit the list at once: numbered thread by thread by a count
  // and a scan, then listed and taken window by window.  (Starts past the list
  // walked where they were found, and contours that meet no line walked by the
  // thread of their first box, left one thread with all levels of a steep edge:
  // 32^2, 1000 levels: 735 us, noise 2220 us; 140 and 228 so.)
  auto windows = [&](auto each, auto take) {
    int n = 0;
    each([&](int, int, int lo, int hi) { n += hi - lo; });
    const int first = block_excl_scan_any<int>(n, &total);
    const int tot = total;
    for (int b = (int)blockIdx.y * TR_SCAP; b < tot; b += (int)gridDim.y * TR_SCAP) {
      int run = first;
      each([&](int m, int y, int lo, int hi) {
        const int z = min(run + hi - lo, b + TR_SCAP);
        for (int s = max(run, b); s < z; s++) slist[s - b] = entry(m, y, lo + 1 + s - run);
        run += hi - lo;
      });
      __syncthreads();
      take(min(TR_SCAP, tot - b));
      __syncthreads();
    }
  };
  auto starts = [&](auto range) {
    tr_starts(T, [&](int m, int y, int c0, int c1, int line, int last) {
      tr_line_starts(m, y, c0, c1, line, last, range);
    }, range);
  };
  if (gridDim.y == 1) {
    auto range = [&](int m, int y, int lo, int hi) {
      int s = atomicAdd(&nstart, hi - lo);
      for (int l = lo + 1; l <= hi && s < TR_SCAP; l++) slist[s++] = entry(m, y, l);
    };
    tr_starts(T, [&](int m, int y, int c0, int c1, int line, int last) {
      tr_line_starts(m, y, c0, c1, line, last, range);
      if (line == 0) nodes += max(0, y ? c0 - c1 : c1 - c0);
      if (line == last) nodes += max(0, y ? c1 - c0 : c0 - c1);
    }, range);
    if (nodes) atomicAdd(&nnode, nodes);
    __syncthreads();
    if (nstart <= TR_SCAP) walk_list(nstart);
    else windows(starts, walk_list);
    if (mine) atomicAdd(&nvis, mine);
    __syncthreads();
    if (nvis == nnode) return;
  } else {
    windows(starts, walk_list);
  }
  // contours that meet no line where chains end: the crossings no chain has
  // taken.  Each is walked from the least of its crossings that move left.
  windows(
      [&](auto range) {
        const int bi = tid >> 1, bj0 = (TY / 2) * (tid & 1);
        for (int j = bj0; j < min(bj0 + TY / 2, th); j++) {
          const int m = (bi + 1) * TS + j;  // entered from the right
          if (C[m] > C[m + 1]) range(m, 0, (int)C[m + 1], (int)C[m]);
        }
      },
      [&](int ns) {
        for (int s = tid; s < ns; s += TR_NT) {
          const int m = (int)(slist[s] >> 17), l = (int)(slist[s] & 0xffffu);
          if (!tr_least(a, T, m, l)) continue;
          const int c = atomicAdd(a.nchain, 1);
          if (c < a.cap) tr_walk(a, T, m, 0, l, c, true);
          else atomicExch(a.err, CASL_ECAPACITY);
        }
      });
}
// CTAs a tile: as many as leave each 4096 crossings, while the tiles alone are
// fewer than the SMs hold.
inline int tr_slices(int ntile, long long ncr) {
  const long long room = 3LL * 148 / ntile, most = ncr / (4096LL * ntile);
  return (int)(room < 2 || most < 2 ? 1 : (room < most ? room : most));
}

// ---------------------------------------------------------------------------
// Positions, in walk layout
// ---------------------------------------------------------------------------
struct PlArgs {
  CrGrid g;
  LevInfo li;
  UField uf;
  ExtGrid eg;
  Consts c;
  const int *off;
  const int2 *own;
  const int4 *R;         // per chain: see k_ch_place
  double *xw, *yw;
  int *cidw;
};
// Position of the crossing of level l on the edge from point (col, row) of the
// tile at (ix0, j0) (congen.f90:211-252, econgen.f90:238-348): the end values
// are the ultra-fine field at the edge's two points, bit for bit the values
// the codes were taken from.
template <bool ECON>
__device__ __forceinline__ double2 tr_place(const PlArgs &a, double qavg, int ix, int r, bool yline, int l) {
  const Consts &c = a.c;
  const int nxu = c.nxu, nyu = c.nyu;
  const double qtmp = qtmp_of(l, a.li);
  if (!yline) {
    if (!ECON) {
      const int iy = r + 1;
      const double q0 = ufield_at(a.uf, qavg, ix, iy, c) - qtmp;
      const double q1 = ufield_at(a.uf, qavg, ix, iy == nyu ? 1 : iy + 1, c) - qtmp;
      const double ygu = c.ymin + c.glyu * (double)(iy - 1);
      const double yy = ygu - c.glyu * q0 / (q1 - q0);
      return make_double2(c.xmin + c.glxu * (double)(ix - 1), c.oms * (yy - c.elly * f_dint(yy * c.hlyi)));
    }
    const int iy = a.eg.iymin + r;
    double q[2];
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const int yy = iy + h, y0 = ext_row0(a.eg, yy, nyu);
      const double v = (yy >= 1 && yy <= nyu)
                           ? ufield_at(a.uf, qavg, ix, yy, c)
                           : ufield_at(a.uf, qavg, ix, y0, c) + a.eg.bfac * (double)(yy - y0);
      q[h] = v - qtmp;
    }
    return make_double2(c.xmin + c.glxu * (double)(ix - 1),
                        (c.glyu * (double)(iy - 1) + c.ymin) - c.glyu * q[0] / (q[1] - q[0]));
  }
  const int ixn = ix == nxu ? 1 : ix + 1;
  const double xgu = c.xmin + c.glxu * (double)(ix - 1);
  double q0, q1, y;
  if (!ECON) {
    const int iy = r + 1;
    q0 = ufield_at(a.uf, qavg, ix, iy, c) - qtmp;
    q1 = ufield_at(a.uf, qavg, ixn, iy, c) - qtmp;
    y = c.ymin + c.glyu * (double)(iy - 1);
  } else {
    const int iy = a.eg.iymin + r, y0 = ext_row0(a.eg, iy, nyu);
    const bool basic = iy >= 1 && iy <= nyu;
    const double qadd = a.eg.bfac * (double)(iy - y0) - qtmp;
    q0 = basic ? ufield_at(a.uf, qavg, ix, iy, c) - qtmp : ufield_at(a.uf, qavg, ix, y0, c) + qadd;
    q1 = basic ? ufield_at(a.uf, qavg, ixn, iy, c) - qtmp : ufield_at(a.uf, qavg, ixn, y0, c) + qadd;
    y = c.glyu * (double)(iy - 1) + c.ymin;
  }
  const double xx = xgu - c.glxu * q0 / (q1 - q0);
  return make_double2(c.oms * (xx - c.ellx * f_dint(xx * c.hlxi)), y);
}
// A tile's own crossings (x-lines of its columns, y-lines of its rows) go
// straight to their places in walk order.  Tile by tile, a contour's
// neighbouring crossings are written close in time, so that the lines of the
// walk arrays fill up in L2; in edge order (all x-lines, then all y-lines)
// the stores alone took 1.1 ms for 25M crossings.  A thread finds its crossed
// edges as bits by packed compares first (looking at every edge in turn: 1.4
// against 1.07 ms).
template <bool ECON>
__global__ void __launch_bounds__(TR_NT) k_tr_place(PlArgs a) {
  CASL_PDL_ENTRY();
  __shared__ __align__(16) unsigned short C[(TX + 1) * TS];
  __shared__ uint2 glist[TR_GCAP];
  __shared__ int wsum[TR_NT / 32], wedge[TR_NT / 32];
  const CrGrid &g = a.g;
  const int tid = threadIdx.x, lane = tid & 31;
  const int ntx = g.nxu / TX;
  const int ix0 = (int)(blockIdx.x % ntx) * TX, j0 = (int)(blockIdx.x / ntx) * TY;
  // The thread's 4 chunks: x-lines of a column (consecutive numbers from id0),
  // or y-lines of 32 columns of two rows (from id0 and id1)
  const bool xl = tid < TX;
  const int col = xl ? tid : 32 * (tid & 3), row = xl ? 0 : ((tid - TX) >> 2) * 2;
  int id0 = 0, id1 = 0, tot = 0;
  if (xl) {
    const long long ch = tr_xchunk(g, ix0, j0, col, 0);
    id0 = __ldg(a.off + ch);
    tot = __ldg(a.off + ch + min(4, g.nseg - (j0 >> 4))) - id0;
  } else {
    const long long c0 = tr_ychunk(g, ix0, j0, row, col >> 4), c1 = tr_ychunk(g, ix0, j0, row + 1, col >> 4);
    if (c0 >= 0) {
      id0 = __ldg(a.off + c0);
      tot += __ldg(a.off + c0 + 2) - id0;
    }
    if (c1 >= 0) {
      id1 = __ldg(a.off + c1);
      tot += __ldg(a.off + c1 + 2) - id1;
    }
  }
  if (!tr_stage(g, ix0, j0, C)) return;
  // the thread's edges with crossings, a bit each: x-lines in order (ma, then
  // mb); y-lines of the first row (ma) and the second (mb)
  unsigned ma = 0, mb = 0;
  const int p0 = col * TS + row;
  if (tot) {
    unsigned w = *reinterpret_cast<const unsigned *>(C + p0);
    if (xl) {
#pragma unroll
      for (int k = 0; k < TY / 2; k++) {
        const unsigned nx = *reinterpret_cast<const unsigned *>(C + p0 + 2 * k + 2);
        const unsigned m = __vcmpne2(w, __funnelshift_r(w, nx, 16)), two = (m & 1u) | (m >> 15 & 2u);
        if (k < 16) ma |= two << (2 * k);
        else mb |= two << (2 * k - 32);
        w = nx;
      }
      const int n = g.ner - j0;  // (a grid open in y may end inside the tile)
      if (n < 32) ma &= (1u << n) - 1u;
      if (n < 64) mb &= n <= 32 ? 0u : (1u << (n - 32)) - 1u;
    } else {
#pragma unroll
      for (int k = 0; k < 32; k++) {
        const unsigned nx = *reinterpret_cast<const unsigned *>(C + p0 + (k + 1) * TS);
        const unsigned m = __vcmpne2(w, nx);
        ma |= (m & 1u) << k;
        mb |= (m >> 31) << k;
        w = nx;
      }
      const int r = j0 + row;
      if (!g.periodic && (r < g.ylo || r >= g.ylo + g.nyl)) ma = 0;
      if (!g.periodic && r + 1 >= g.ylo + g.nyl) mb = 0;
    }
  }
  const int ne = __popc(ma) + __popc(mb);
  const int incl = warp_incl_scan(tot), eincl = warp_incl_scan(ne);
  if (lane == 31) {
    wsum[tid >> 5] = incl;
    wedge[tid >> 5] = eincl;
  }
  __syncthreads();
  int s0 = incl - tot, all = 0, e0 = eincl - ne, edges = 0;
  for (int w = 0; w < TR_NT / 32; w++) {
    if (w < tid >> 5) {
      s0 += wsum[w];
      e0 += wedge[w];
    }
    all += wsum[w];
    edges += wedge[w];
  }
  const double qavg = ufield_qavg(a.uf.lsum, a.uf.qjump, a.uf.have, a.c.nxu, a.c.nyu);
  // the thread's edges in order: f(point, first number, lower code, crossings)
  auto each_edge = [&](auto f) {
    int id = id0;
#pragma unroll
    for (int h = 0; h < 2; h++) {
      if (!xl && h) id = id1;
      for (unsigned m = h ? mb : ma; m; m &= m - 1) {
        const int k = __ffs(m) - 1;
        const int p = xl ? p0 + 32 * h + k : p0 + h + k * TS;
        const int c0 = C[p], c1 = C[p + (xl ? 1 : TS)], n = abs(c1 - c0);
        f((unsigned)(p << 1 | !xl) << 16, id, min(c0, c1), n);
        id += n;
      }
    }
  };
  auto put = [&](unsigned e, int id) {  // edge << 16 | level
    const int2 o = __ldg(&a.own[id]);
    const int4 R = __ldg(&a.R[o.x]);
    const int m = (int)(e >> 17), cx = tr_col(m), cy = m - cx * TS;
    const double2 v = tr_place<ECON>(a, qavg, ix0 + cx + 1, j0 + cy, (e >> 16) & 1u, (int)(e & 0xffffu));
    if (R.w < 0) return;
    int rp = R.x + o.y;
    if (rp < 0) rp += R.y;
    const long long pos = (long long)R.z + rp;
    a.xw[pos] = v.x;
    a.yw[pos] = v.y;
    a.cidw[pos] = R.w;  // the contour of every walk position, for the first renode
  };
  if (all <= TR_MANY * edges) {
    for (int b = (int)blockIdx.y * TR_GCAP; b < all; b += (int)gridDim.y * TR_GCAP) {
      if (tot && s0 < b + TR_GCAP && s0 + tot > b) {
        int s = s0;
        each_edge([&](unsigned e, int id, int lo, int n) {
          for (int l = lo + 1; l <= lo + n; l++, s++, id++)
            if (s >= b && s < b + TR_GCAP) glist[s - b] = make_uint2(e | (unsigned)l, (unsigned)id);
        });
      }
      __syncthreads();
      for (int s = tid; s < min(TR_GCAP, all - b); s += TR_NT) put(glist[s].x, (int)glist[s].y);
      __syncthreads();
    }
    return;
  }
  // Many levels an edge: the edges are listed, with the places of their first
  // crossings, and a crossing finds its edge by search.  (A thread that lists
  // its crossings one by one fills whole batches alone: 32^2, 1000 levels, with
  // a CTA a tile, 2.0 ms, and 0.2 so.)
  constexpr int EC = TR_GCAP / 2;
  int *gst = reinterpret_cast<int *>(glist + EC);  // EC + 1 of them
  for (int b = 0; b < edges; b += EC - 1) {
    const int nl = min(EC - 1, edges - b);
    if (ne && e0 < b + nl && e0 + ne > b) {
      int s = s0, q = e0 - b;
      each_edge([&](unsigned e, int id, int lo, int n) {
        if (q >= 0 && q < nl) {
          glist[q] = make_uint2(e | (unsigned)lo, (unsigned)id);
          gst[q] = s;
          if (q == nl - 1) gst[nl] = s + n;
        }
        s += n;
        q++;
      });
    }
    __syncthreads();
    const int end = gst[nl];
    for (int s = gst[0] + (int)blockIdx.y * TR_NT + tid; s < end; s += (int)gridDim.y * TR_NT) {
      int lo = 0, hi = nl;  // gst[lo] <= s < gst[hi]
      while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (gst[mid] <= s) lo = mid; else hi = mid;
      }
      const int k = s - gst[lo];
      put(glist[lo].x + 1u + (unsigned)k, (int)glist[lo].y + k);
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// Ranking over the chains
// ---------------------------------------------------------------------------
// Each chain's jump state is one 16-byte record (next, minimum, terminal flag),
// one gather a hop.  A launch makes three hops (windows grow fourfold): at a few
// hundred thousand chains it is the launches and the gathers' latency that
// cost, not the bytes.  The last chain of a list is its own next, so next ends
// there in the launch that sets the flag; around a cycle it keeps turning and
// says nothing.  A launch that changes no minimum and no flag leaves none to
// change (a window that does not cover its cycle has a chain whose minimum the
// next one lowers, one that does not reach its list's end a chain whose flag it
// sets), so the launches after it return at once: flag[it] says whether launch
// it changed anything.
__global__ void k_ch_init(const int4 *__restrict__ chain, const int2 *__restrict__ own, int S,
                          int *__restrict__ nexts, int4 *__restrict__ J, int *__restrict__ err) {
  CASL_PDL_ENTRY();
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < S; k += gridDim.x * blockDim.x) {
    const int4 c = chain[k];
    int n = c.x < 0 ? -1 : own[c.x].x;
    if (n >= S || n < -1) {
      atomicExch(err, CASL_EINVAL);
      n = -1;
    }
    nexts[k] = n;
    J[k] = make_int4(n < 0 ? k : n, c.z, n < 0, 0);
  }
}
__global__ void k_ch_jump1(const int4 *__restrict__ J, int S, int4 *__restrict__ J2, int it,
                           int *__restrict__ flag) {
  CASL_PDL_ENTRY();
  if (it > 0 && flag[it - 1] == 0) return;
  bool changed = false;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < S; k += gridDim.x * blockDim.x) {
    const int4 a = J[k];
    int4 r = a;
#pragma unroll
    for (int h = 0; h < 3; h++) {
      const int4 b = J[r.x];
      r = make_int4(b.x, min(r.y, b.y), r.z | b.z, 0);
    }
    J2[k] = r;
    changed |= r.y != a.y || r.z != a.z;
  }
  if (__syncthreads_or(changed) && threadIdx.x == 0 && __ldcg(flag + it) == 0) flag[it] = 1;
}
// (link, suffix sum) of the suffix-sum jumps, one 16-byte record
struct __align__(16) SlSuf {
  long long suf;
  int sl, pad;
};
// List for the suffix sums: a cycle is cut before the chain that holds its
// least crossing (its head); other lists end at their last chain.
__global__ void k_ch_list(const int *__restrict__ nexts, const int4 *__restrict__ J,
                          const int2 *__restrict__ own, const int4 *__restrict__ chain, int S,
                          SlSuf *__restrict__ L, int *__restrict__ head) {
  CASL_PDL_ENTRY();
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < S; k += gridDim.x * blockDim.x) {
    const int4 j = J[k];
    const int n = nexts[k];
    const int h = j.z ? -1 : own[j.y].x;
    head[k] = h;
    L[k] = SlSuf{(long long)chain[k].y, h >= 0 && n == h ? -1 : n, 0};
  }
}
__global__ void k_ch_jump2(const SlSuf *__restrict__ L, int S, SlSuf *__restrict__ L2, int it,
                           int *__restrict__ flag) {
  CASL_PDL_ENTRY();
  if (it > 0 && flag[it - 1] == 0) return;
  bool changed = false;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < S; k += gridDim.x * blockDim.x) {
    SlSuf a = L[k];
    changed |= a.sl >= 0;
#pragma unroll
    for (int h = 0; h < 3; h++)
      if (a.sl >= 0) {
        const SlSuf b = L[a.sl];
        a = SlSuf{a.suf + b.suf, b.sl, 0};
      }
    L2[k] = a;
  }
  if (__syncthreads_or(changed) && threadIdx.x == 0 && __ldcg(flag + it) == 0) flag[it] = 1;
}
// The closed contours: one slot per cycle, in any order; the key sorts them
// by level and least crossing.
__global__ void k_ch_heads(const int *__restrict__ head, const int4 *__restrict__ J,
                           const SlSuf *__restrict__ L, const int *__restrict__ clev, int S,
                           unsigned long long *__restrict__ key, int *__restrict__ slot,
                           int *__restrict__ len, int *__restrict__ cslot, int *__restrict__ nc) {
  CASL_PDL_ENTRY();
  for (int b = blockIdx.x * blockDim.x; b < S; b += gridDim.x * blockDim.x) {
    const int k = b + threadIdx.x, lane = threadIdx.x & 31;
    const bool f = k < S && head[k] == k;
    const unsigned m = __ballot_sync(0xffffffffu, f);
    int at = 0;
    if (lane == 0 && m) at = atomicAdd(nc, __popc(m));
    at = __shfl_sync(0xffffffffu, at, 0) + __popc(m & ((1u << lane) - 1u));
    if (f) {
      key[at] = (unsigned long long)(unsigned)clev[k] << 32 | (unsigned)J[k].y;
      slot[at] = at;
      len[at] = (int)L[k].suf;
      cslot[k] = at;
    }
  }
}
// At the crossings st[0..m): the last crossing of their list, its length from
// there on, its least crossing, the length from that one on, the level and
// the list's last chain.
__global__ void k_ch_query(const int *__restrict__ st, int m, const int2 *__restrict__ own,
                           const int4 *__restrict__ J, const SlSuf *__restrict__ L,
                           const int4 *__restrict__ chain, const int *__restrict__ clev,
                           int *__restrict__ out) {
  CASL_PDL_ENTRY();
  for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < m; q += gridDim.x * blockDim.x) {
    const int2 o = own[st[q]];
    const int4 j = J[o.x];
    const int2 om = own[j.y];
    out[q] = chain[j.x].w;
    out[m + q] = (int)L[o.x].suf - o.y;
    out[2 * m + q] = j.y;
    out[3 * m + q] = (int)L[om.x].suf - om.y;
    out[4 * m + q] = clev[o.x];
    out[5 * m + q] = j.x;
  }
}
// Contours in order: lengths, levels, and each slot's place.
__global__ void k_ct_order(const unsigned long long *__restrict__ key, const int *__restrict__ slot,
                           const int *__restrict__ len, int C, int nlevm, int *__restrict__ clen,
                           int *__restrict__ clevt, int *__restrict__ place) {
  CASL_PDL_ENTRY();
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < C; j += gridDim.x * blockDim.x) {
    const int s = slot[j], lev = (int)(key[j] >> 32);
    clen[j] = len[s];
    clevt[j] = lev - nlevm + (lev - 1) / nlevm - 1;
    place[s] = j;
  }
}
// Per chain: place p of the chain lies at coff + (r + p), plus the contour's
// length where r + p is negative: (r, length, coff, contour).  Chains of lists
// that end (between saddles) take the host's placement of their list.
__global__ void k_ch_place(const int *__restrict__ head, const int4 *__restrict__ J,
                           const SlSuf *__restrict__ L, const int2 *__restrict__ own,
                           const int *__restrict__ cslot, const int *__restrict__ place,
                           const int *__restrict__ coff, const int *__restrict__ clen,
                           const int *__restrict__ listof, const int *__restrict__ ladd,
                           const int *__restrict__ lslot, int S, int4 *__restrict__ R) {
  CASL_PDL_ENTRY();
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < S; k += gridDim.x * blockDim.x) {
    const int h = head[k];
    const int suf = (int)L[k].suf;
    if (h >= 0) {
      const int c = place[cslot[h]], len = clen[c];
      R[k] = make_int4(len - suf - own[J[k].y].y, len, coff[c], c);
    } else {
      const int q = listof ? listof[J[k].x] : -1;
      if (q < 0) {
        R[k] = make_int4(0, 0, 0, -1);
      } else {
        const int c = place[lslot[q]];
        R[k] = make_int4(ladd[q] - suf, clen[c], coff[c], c);
      }
    }
  }
}
__global__ void k_list_of(const int *__restrict__ last, int m, int *__restrict__ listof) {
  CASL_PDL_ENTRY();
  for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < m; q += gridDim.x * blockDim.x)
    listof[last[q]] = q;
}
}  // namespace casl

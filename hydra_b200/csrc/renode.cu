// Parallel renode of many contours (contours.f90:687-933); see renode.cuh.
#include <math.h>

#include <algorithm>

#include "renode.cuh"

namespace casl {

__device__ __forceinline__ long long wnext(long long w, long long cs, long long L) {
  return w + 1 < cs + L ? w + 1 : cs;
}
__device__ __forceinline__ long long wprev(long long w, long long cs, long long L) {
  return w > cs ? w - 1 : cs + L - 1;
}

__global__ void __launch_bounds__(256) k_rn_cid(RenodeIn in, long long N, int *__restrict__ cid) {
  CASL_PDL_ENTRY();
  const int C = contours_in(in);
  for (long long b = blockIdx.x * (long long)CC_CHUNK; b < N; b += (long long)gridDim.x * CC_CHUNK) {
    chunk_contours(in.cs, C, b);
    for (long long w = b + threadIdx.x; w < min(N, b + CC_CHUNK); w += blockDim.x)
      cid[w] = chunk_contour_of(in.cs, C, w);
  }
}

// The node densities of renode (contours.f90:718-796) for node w: dx, dy,
// |d| to the next node; corners and curvature b; spherical-curvature
// densities; node curvature as a weighted average; the fractional node count.
// Only the density e and the corner flag are kept (the placement forms the
// cubic of a segment again where it puts nodes).  rn_node recomputes every
// quantity node w needs from the coordinates of nodes w-2..w+3 (cyclic in the
// contour); k_rn_nodes computes each quantity once per node and passes it to
// the neighbouring lanes, with rn_node for the warps whose nodes come near a
// contour's end.  Both use the same expressions in the same order.
__device__ __forceinline__ void rn_node(const RenodeIn &in, const RenodeScratch &s, const Consts &c,
                                        long long w, double &eout, int &cout) {
  const int k = s.cid[w];
  const long long cs = in.cs[k], L = in.len[k];
  long long j[6];
  j[2] = w;
  j[1] = wprev(w, cs, L);
  j[0] = wprev(j[1], cs, L);
  j[3] = wnext(w, cs, L);
  j[4] = wnext(j[3], cs, L);
  j[5] = wnext(j[4], cs, L);
  double X[6], Y[6];
#pragma unroll
  for (int m = 0; m < 6; m++) {
    X[m] = in.xw[j[m]];
    Y[m] = in.yw[j[m]];
  }
  // rn1 at nodes m = 0..4
  double dx[5], dy[5], v[5], e1[5];
#pragma unroll
  for (int m = 0; m < 5; m++) {
    double xx = X[m + 1] - X[m];
    dx[m] = xx - c.ellx * f_dint(xx * c.hlxi);
    double yy = Y[m + 1] - Y[m];
    dy[m] = yy - c.elly * f_dint(yy * c.hlyi);
    v[m] = dx[m] * dx[m] + dy[m] * dy[m];
    e1[m] = sqrt(v[m]);
  }
  // rn2 at nodes m = 1..4
  double b[5];
  int corner2 = 0;
#pragma unroll
  for (int m = 1; m < 5; m++) {
    double u = v[m - 1], a = -dx[m - 1], cc = -dy[m - 1];
    int corner = dx[m] * a + dy[m] * cc > 0.0;
    if (m == 2) corner2 = corner;
    if (corner) {
      b[m] = 0.0;
    } else {
      double t1 = a * v[m] - dx[m] * u, t2 = cc * v[m] - dy[m] * u;
      b[m] = (dx[m] * cc - a * dy[m]) / sqrt(t1 * t1 + t2 * t2 + c.small3);
    }
  }
  // rn3 at nodes m = 1..3
  double u2[4], v2[4];
#pragma unroll
  for (int m = 1; m < 4; m++) {
    double u = e1[m] * (b[m + 1] + b[m]);
    double ww = 1.0 / (v[m] + c.dmsq);
    u2[m] = ww * sqrt(c.elf * v[m] + u * u);
    v2[m] = ww * e1[m];
  }
  // rn4 at nodes 2, 3 and rn5 at node 2
  const double d2 = (u2[1] + u2[2]) / (v2[1] + v2[2] + c.small);
  const double d3 = (u2[2] + u2[3]) / (v2[2] + v2[3] + c.small);
  const double uu = 0.5 * (d2 + d3);
  const double t = c.densf * sqrt(uu) + uu;
  s.e[w] = eout = e1[2] * fmin(c.dmi, t);
  cout = corner2;
  if (corner2) red_add_s32(&s.ccnt[k], 1);
}

// Densities, their sums along each contour and the corners' ranks, in one
// pass: a tile of RN_IT x 224 nodes per block.
//
// One warp covers nodes base-2 .. base+29 (lane L holds node base-2+L) and
// writes nodes base .. base+27 (lanes 2..29): the segment quantities (rn1)
// of lane L, its curvature (rn2), its cubic and density terms (rn3) and its
// rn4 average each take the lower neighbour's value from lane L-1 and the
// upper neighbour's from lane L+1.  Valid while every written node's
// stencil w-2..w+3 lies inside its contour without wrapping, which the first
// and last node of the warp's stencils tell (a contour's nodes are
// consecutive); otherwise the warp takes rn_node.
//
// The densities and flags stay in shared memory for the tile's scans; tiles
// look back at earlier ones for the corners before them (any order: integers)
// and, to the last contour start before the tile, for the densities, whose
// tile sums are added from left to right (the same on every run).
//
// Bound by the latency of a step's chain (three square roots and three
// divisions one after the other, 24 warps an SM): the next step's nodes are
// loaded before it, and the sums and ranks leave through shared memory (a
// thread's 7 consecutive nodes would write 4 sectors for 1).  24M nodes 1036 us
// before, with the cubic's five coefficients stored as well, and 630 so.
constexpr int RN_OUT = 28, RN_WARPS = 8, RN_STEP = RN_OUT * RN_WARPS;
template <int RN_IT>
__global__ void __launch_bounds__(256, 3) k_rn_nodes(RenodeIn in, RenodeScratch s, Consts c) {
  CASL_PDL_ENTRY();
  const unsigned FULL = 0xffffffffu;
  constexpr int RN_TILE = RN_STEP * RN_IT;
  __shared__ double te[RN_TILE];
  __shared__ int tc[RN_TILE];
  __shared__ unsigned char tf[RN_TILE];  // 1: contour start, 2: corner
  __shared__ SegPair total;
  __shared__ unsigned int ctot, cbefore;
  __shared__ double carry;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const long long N = in.N;
  const int tile = lb_ticket(&s.tick[0]);
  const long long t0 = (long long)tile * RN_TILE;
  if (t0 >= N) return;
  // this lane's node of a step and, in lane 31, the one after: coordinates, contours
  double pX, pY, pX1, pY1;
  int pk, pk1;
  auto fetch = [&](int it) {
    const long long o = t0 + (long long)(it * RN_WARPS + wid) * RN_OUT - 2 + lane;
    pX = pY = pX1 = pY1 = 0.0;
    pk = pk1 = 0;
    if (o >= 0 && o < N) {
      pX = in.xw[o];
      pY = in.yw[o];
      pk = s.cid[o];
    }
    if (lane == 31 && o + 1 < N) {
      pX1 = in.xw[o + 1];
      pY1 = in.yw[o + 1];
      pk1 = s.cid[o + 1];
    }
  };
  fetch(0);
#pragma unroll 1
  for (int it = 0; it < RN_IT; it++) {
    const long long base = t0 + (long long)(it * RN_WARPS + wid) * RN_OUT;
    if (base >= N) break;
    const double X = pX, Y = pY, X1 = pX1, Y1 = pY1;
    const int k = pk, k1 = pk1;
    if (it + 1 < RN_IT) fetch(it + 1);
    const long long o = base - 2 + lane;  // this lane's node
    const bool out = lane >= 2 && lane < 2 + RN_OUT && o < N;
    double e = 0.0;
    int corner = 0;
    const int kf = __shfl_sync(FULL, k, 0), kl = __shfl_sync(FULL, k1, 31);
    if (base < 2 || base + RN_OUT + 2 >= N || kf != kl) {
      if (out) {
        rn_node(in, s, c, o, e, corner);
        te[o - t0] = e;
        tf[o - t0] = (unsigned char)((o == in.cs[k]) | corner << 1);
      }
      continue;
    }
    double Xn = __shfl_down_sync(FULL, X, 1), Yn = __shfl_down_sync(FULL, Y, 1);
    if (lane == 31) {
      Xn = X1;
      Yn = Y1;
    }
    // rn1: the segment to the next node
    const double xx = Xn - X;
    const double dx = xx - c.ellx * f_dint(xx * c.hlxi);
    const double yy = Yn - Y;
    const double dy = yy - c.elly * f_dint(yy * c.hlyi);
    const double v = dx * dx + dy * dy;
    const double e1 = sqrt(v);
    // rn2 at this node, from the previous segment
    const double up = __shfl_up_sync(FULL, v, 1);
    const double a = -__shfl_up_sync(FULL, dx, 1), ccp = -__shfl_up_sync(FULL, dy, 1);
    corner = dx * a + dy * ccp > 0.0;
    double b;
    if (corner) {
      b = 0.0;
    } else {
      const double t1 = a * v - dx * up, t2 = ccp * v - dy * up;
      b = (dx * ccp - a * dy) / sqrt(t1 * t1 + t2 * t2 + c.small3);
    }
    // rn3 at this node, with the next node's curvature
    const double bn = __shfl_down_sync(FULL, b, 1);
    const double u = e1 * (bn + b);
    const double ww = 1.0 / (v + c.dmsq);
    const double u2 = ww * sqrt(c.elf * v + u * u);
    const double v2 = ww * e1;
    // rn4 at this node (with the previous node's rn3) and at the next one
    const double u2p = __shfl_up_sync(FULL, u2, 1), v2p = __shfl_up_sync(FULL, v2, 1);
    const double d = (u2p + u2) / (v2p + v2 + c.small);
    const double dn = __shfl_down_sync(FULL, d, 1);
    if (out) {
      // rn5
      const double uu = 0.5 * (d + dn);
      const double t = c.densf * sqrt(uu) + uu;
      e = e1 * fmin(c.dmi, t);
      s.e[o] = e;
      te[o - t0] = e;
      tf[o - t0] = (unsigned char)(corner << 1);
      if (corner) red_add_s32(&s.ccnt[k], 1);
    }
  }
  __syncthreads();
  // the tile's scans, PT nodes per thread
  constexpr int PT = (RN_TILE + 255) / 256;
  const int n = (int)min((long long)RN_TILE, N - t0), i0 = PT * threadIdx.x;
  SegPair acc{0.0, 0};
  int nc = 0;
#pragma unroll
  for (int q = 0; q < PT; q++)
    if (i0 + q < n) {
      acc = seg_op(acc, SegPair{te[i0 + q], tf[i0 + q] & 1});
      nc += tf[i0 + q] >> 1;
    }
  SegPair run = block_seg_excl(acc, &total);
  const unsigned int before = block_excl_scan_any<unsigned int>((unsigned)nc, &ctot);
  if (wid == 0) {
    if (lane == 0) {
      s.tilev[tile] = total.v;
      s.tilef[tile] = total.f;
      __threadfence();
    }
    __syncwarp();
    const unsigned long long pre = lb_prefix(s.nstat, tile, ctot, s.err);
    if (lane == 0) cbefore = (unsigned)pre;
    // The densities from the last contour start up to this tile.  Every tile
    // whose sum is needed has published it before its status word; one that
    // the corners' look-back did not reach is waited for here.
    auto ready = [&](int t) {
      const long long c0 = clock64();
      while (lb_load(&s.nstat[t]) == 0)
        if (clock64() - c0 > 2000000000LL) {
          atomicExch(s.err, CASL_ETIMEOUT);
          break;
        }
    };
    double v = 0.0;
    if (tile > 0 && !(tf[0] & 1)) {
      int j = tile - 1;  // the tile of that start
      for (;; j -= 32) {
        const int t = j - lane;
        bool f = t <= 0;
        if (t >= 0) {
          ready(t);
          f = f || __ldcg(&s.tilef[t]) != 0;
        }
        const unsigned m = __ballot_sync(FULL, f);
        if (m) {
          j -= __ffs(m) - 1;
          break;
        }
      }
      j = max(j, 0);
      for (; j < tile; j += 32) {
        const int t = j + lane;
        const double x = t < tile ? __ldcg(&s.tilev[t]) : 0.0;
        for (int q = 0; q < min(32, tile - j); q++) v = v + __shfl_sync(FULL, x, q);
      }
    }
    if (lane == 0) carry = v;
  }
  __syncthreads();
  int rank = (int)(cbefore + before);
#pragma unroll
  for (int q = 0; q < PT; q++)
    if (i0 + q < n) {
      const int f = tf[i0 + q];
      run = seg_op(run, SegPair{te[i0 + q], f & 1});
      te[i0 + q] = run.f ? run.v : run.v + carry;
      tc[i0 + q] = 2 * rank + (f >> 1);
      if (f & 2) s.cornerpos[rank++] = (int)(t0 + i0 + q);
    }
  __syncthreads();
  for (int i = threadIdx.x; i < n; i += 256) {
    s.S[t0 + i] = te[i];
    s.cc[t0 + i] = tc[i];
  }
}

// Sum of e over `m` nodes of contour [cs, cs+L) starting at walk index st.
__device__ __forceinline__ double sumrange(const double *__restrict__ S, long long cs,
                                           long long L, long long st, long long m) {
  long long a = st - cs, b = a + m;
  auto pre = [&](long long k) -> double { return k == 0 ? 0.0 : S[cs + k - 1]; };
  if (b <= L) return pre(b) - pre(a);
  return (pre(L) - pre(a)) + pre(b - L);
}

__device__ __forceinline__ int nint_d(double x) { return (int)llround(x); }

// The reference adds a contour's (or a corner piece's) densities one after
// the other from its first node (contours.f90:799-806, 843-853) and rounds
// the total to the node count.  The prefix sums here group the additions
// otherwise; where the total lies within 1e-6 of a half-integer, so that
// the grouping could move it across the rounding point, it is recomputed in
// the reference's order: m densities from node st, wrapping within
// [cs, cs+L).
__device__ __forceinline__ bool near_half(double x) {
  const double f = x - floor(x);
  return fabs(f - 0.5) < 1e-6;
}
__device__ double seq_sum(const double *__restrict__ e, long long cs, long long L, long long st,
                          long long m) {
  double t = 0.0;
  long long i = st - cs;
  for (long long j = 0; j < m; j++) {
    t = t + e[cs + i];
    if (++i == L) i = 0;
  }
  return t;
}

// A contour's pieces (contours.f90:799-809, 813-930): its nodes, corners, density
// total, first corner and first piece.
struct RnContour {
  long long cs, L;
  double total;
  int nc, np, cfirst, p0;
};
// Piece q of it, stored; its new nodes.
__device__ __forceinline__ int rn_piece(const RenodeScratch &s, const Consts &c, const RnContour &a,
                                        int q) {
  long long st, pl;
  double sum;
  int n;
  if (a.nc <= 1) {
    st = a.nc == 0 ? a.cs : s.cornerpos[a.cfirst];
    pl = a.L;
    sum = a.total;
    n = nint_d(a.total) + 1;
  } else {
    st = s.cornerpos[a.cfirst + q];
    const long long en = s.cornerpos[a.cfirst + (q + 1) % a.nc];
    pl = en - st;  // both corners lie in [cs, cs+L)
    if (pl < 0) pl += a.L;
    sum = sumrange(s.S, a.cs, a.L, st, pl);
    if (near_half(sum)) sum = seq_sum(s.e, a.cs, a.L, st, pl);
    n = sum > c.small ? nint_d(sum) + 1 : 0;
  }
  const double preA = st == a.cs ? 0.0 : s.S[st - 1];
  s.piece[a.p0 + q] = RnPiece{(int)st, (int)pl, n, 0, n > 0 ? (double)n / sum : 0.0,
                              preA, s.S[a.cs + a.L - 1] - preA, 0.0};
  return n;
}

// Per contour: node count and pieces, and where its nodes go in the output:
// tiles of 256 contours, whose kept nodes and contours are scanned by looking
// back (packed as nodes * 2^31 + contours).  Pieces are stored block by block
// from a running total; their order is free.  Contours of more than RN_MANY
// pieces are taken by the whole block: a thread alone needs half a
// microsecond a corner, which the tiles behind it wait for (one contour of
// 200,000 corners 107 ms, 1.8 so; from two million on those waits ran out).
constexpr int RN_MANY = 64;
__global__ void __launch_bounds__(256) k_rn_contours(RenodeIn in, RenodeScratch s, RenodeOut out,
                                                     Consts c, int mode) {
  CASL_PDL_ENTRY();
  __shared__ int ptot, pbase, nmany;
  __shared__ unsigned long long ntot, nbefore;
  __shared__ int many[256], mn[256];  // the tile's long contours; their new nodes, then outputs
  __shared__ RnContour mc[256];
  const int Ce = contours_in(in), ntile = (Ce + 255) / 256, tid = threadIdx.x;
  while (true) {
    const int tile = lb_ticket(&s.tick[1]);
    if (tile >= ntile) {
      if (ntile == 0 && tile == 0 && tid < 3) out.d_counts[tid] = 0;
      return;
    }
    if (tid == 0) nmany = 0;
    const int k = tile * 256 + tid;
    RnContour a{};
    if (k < Ce) {
      a.cs = in.cs[k];
      a.L = in.len[k];
      a.nc = s.ccnt[k];
      a.total = s.S[a.cs + a.L - 1];
      if (near_half(a.total)) a.total = seq_sum(s.e, a.cs, a.L, a.cs, a.L);
      if (!(mode == RENODE_SURGERY && a.L <= 3)) {
        int npr0 = nint_d(a.total) + 1;
        if (npr0 >= 3) a.np = a.nc > 1 ? a.nc : 1;
      }
    }
    const int ex = block_excl_scan_any<int>(a.np, &ptot);
    if (tid == 0) pbase = ptot ? atomicAdd(&s.tick[2], ptot) : 0;
    __syncthreads();
    a.p0 = pbase + ex;
    a.cfirst = a.np ? s.cc[a.cs] >> 1 : 0;
    int npr = 0;
    if (a.np > RN_MANY) {
      many[atomicAdd(&nmany, 1)] = tid;
      mc[tid] = a;
    } else {
      for (int q = 0; q < a.np; q++) npr += rn_piece(s, c, a, q);
    }
    __syncthreads();
    for (int m = 0; m < nmany; m++) {
      const RnContour b = mc[many[m]];
      int n = 0;
      for (int q = tid; q < b.np; q += 256) n += rn_piece(s, c, b, q);
      block_excl_scan_any<int>(n, &ptot);
      if (tid == many[m]) npr = ptot;
      __syncthreads();
    }
    const bool keep = k < Ce && (mode == RENODE_SURGERY ? npr > 3 : npr > 0);
    const unsigned long long mine = keep ? ((unsigned long long)npr << 31) + 1ull : 0ull;
    unsigned long long at = block_excl_scan_any<unsigned long long>(mine, &ntot);
    if (tid < 32) {
      const unsigned long long pre = lb_prefix(s.cstat, tile, ntot, s.err);
      if (tid == 0) nbefore = pre;
    }
    __syncthreads();
    at += nbefore;
    mn[tid] = -1;
    if (k < Ce) {
      s.poff[k] = keep ? a.p0 : -1;
      if (keep) {
        int base = (int)(at >> 31);
        const int j = (int)(at & 0x7fffffffull);
        out.ocs[j] = base;
        out.olen[j] = npr;
        out.olev[j] = in.levt ? in.levt[k] : 0;
        if (a.np > RN_MANY) {
          mn[tid] = base;
        } else {
          for (int q = 0; q < a.np; q++) {
            s.piece[a.p0 + q].out = base;
            base += s.piece[a.p0 + q].n;
          }
        }
      }
    }
    __syncthreads();
    for (int m = 0; m < nmany; m++) {
      int base = mn[many[m]];
      if (base < 0) continue;
      const int np = mc[many[m]].np;
      RnPiece *p = s.piece + mc[many[m]].p0;
      for (int q0 = 0; q0 < np; q0 += 256) {
        const int q = q0 + tid;
        const int off = block_excl_scan_any<int>(q < np ? p[q].n : 0, &ptot);
        if (q < np) p[q].out = base + off;
        base += ptot;
        __syncthreads();
      }
    }
    if (tile == ntile - 1 && tid == 0) {
      const unsigned long long all = nbefore + ntot;
      const long long nodes = (long long)(all >> 31);
      out.d_counts[0] = (int)(all & 0x7fffffffull);
      out.d_counts[1] = (int)nodes;
      out.d_counts[2] = nodes > out.cap;
    }
  }
}

// The new nodes: node t of a piece lies on the old segment whose cumulative
// density reaches t (contours.f90:856-928).
//
// A block takes 128 * PU consecutive nodes.  First each one's cumulative
// densities Ep, Ec at its two ends (in units of new nodes) say whether its
// segment receives any; those that do (one in 18 of a recontouring's crossings,
// most nodes of a state) are gathered in shared memory, so that the second half
// runs on full warps: the segment's cubic from its four nodes, and the nodes.
// A warp whose nodes lie in one piece of a contour, the usual case, reads its
// data once and per node only the prefix sum.  24M crossings: 684 us with a
// node a thread and its contour's data loaded for each, 287 so; 1.4M nodes 52
// both ways.
constexpr int PL_BT = 128;
template <int PU>
__global__ void __launch_bounds__(PL_BT, 8) k_rn_place(RenodeIn in, RenodeScratch s, RenodeOut out,
                                                  Consts c) {
  CASL_PDL_ENTRY();
  if (out.d_counts[2]) return;  // overflow: the caller reports it
  constexpr int TILE = PL_BT * PU;
  __shared__ double lEp[TILE], lEc[TILE];
  __shared__ int lw[TILE], lp[TILE];
  __shared__ int nl;
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const double f12 = 0.5, f13 = 1.0 / 3.0, f16 = 1.0 / 6.0;
  for (long long b = blockIdx.x * (long long)TILE; b < in.N; b += (long long)gridDim.x * TILE) {
    __syncthreads();  // the list of the tile before is done with
    if (threadIdx.x == 0) nl = 0;
    __syncthreads();
    const long long wb = b + wid * 32 * PU, we = min(wb + 32 * PU, in.N) - 1;
    if (wb <= we) {
      double S[PU];
#pragma unroll
      for (int u = 0; u < PU; u++) S[u] = wb + 32 * u + lane <= we ? s.S[wb + 32 * u + lane] : 0.0;
      double last = wb > 0 ? s.S[wb - 1] : 0.0;  // the sum before the warp's next 32 nodes
      // the piece of node w of contour k, whose first node is cs (-1: not kept)
      auto piece_of = [&](long long w, int k, long long cs) -> int {
        const int nc = s.ccnt[k], p0 = s.poff[k];
        if (nc < 2 || p0 < 0) return p0;
        const int cw = s.cc[w];
        const int q = (cw >> 1) - (s.cc[cs] >> 1) + (cw & 1) - 1;
        return p0 + (q < 0 ? nc - 1 : q);
      };
      int k = s.cid[wb], p = -1;
      long long cs = in.cs[k];
      RnPiece pc{};
      bool one = k == s.cid[we];
      if (one) {
        // the same piece at both ends, and both before or both after its
        // first node (the last piece wraps), is the same between them
        p = piece_of(wb, k, cs);
        one = p == piece_of(we, k, cs);
        if (one && p >= 0) {
          pc = s.piece[p];
          one = (wb < pc.st) == (we < pc.st);
        }
      }
#pragma unroll
      for (int u = 0; u < PU; u++) {
        const long long w = wb + 32 * u + lane;
        double P0 = __shfl_up_sync(FULL, S[u], 1);
        if (lane == 0) P0 = last;
        last = __shfl_sync(FULL, S[u], 31);
        if (!one) {
          p = -1;
          if (w <= we) {
            k = s.cid[w];
            cs = in.cs[k];
            p = piece_of(w, k, cs);
            if (p >= 0) pc = s.piece[p];
          }
        }
        int pw = w <= we ? p : -1;  // the node's piece, when it receives nodes
        double Ep = 0.0, Ec = 0.0;
        if (pw >= 0 && pc.n == 0) pw = -1;
        if (pw >= 0) {
          // sums of the piece's densities before and through w (sumrange's
          // two cases, which agree where a range ends at the contour's end)
          if (w == cs) P0 = 0.0;
          Ep = pc.fac * (w < pc.st ? pc.preW + P0 : P0 - pc.preA);
          Ec = pc.fac * (w < pc.st ? pc.preW + S[u] : S[u] - pc.preA);
          if (w == pc.st) {
            out.xo[pc.out] = in.xw[w];
            out.yo[pc.out] = in.yw[w];
          }
        }
        if (pw >= 0) {
          long long t0 = (long long)floor(Ep) + 1, t1 = (long long)floor(Ec);
          if (t1 > pc.n - 1) t1 = pc.n - 1;
          if (t0 < 1) t0 = 1;
          if (t1 < t0) pw = -1;
        }
        const unsigned m = __ballot_sync(FULL, pw >= 0);
        if (m) {
          int at = 0;
          if (lane == 0) at = atomicAdd(&nl, __popc(m));
          at = __shfl_sync(FULL, at, 0) + __popc(m & ((1u << lane) - 1u));
          if (pw >= 0) {
            lw[at] = (int)w;
            lp[at] = pw;
            lEp[at] = Ep;
            lEc[at] = Ec;
          }
        }
      }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < nl; i += PL_BT) {
      const long long w = lw[i];
      const int k = s.cid[w];
      const RnPiece &pc = s.piece[lp[i]];
      const int n = pc.n;
      const long long cs = in.cs[k], L = in.len[k], o = pc.out;
      const double Ep = lEp[i], Ec = lEc[i];
      const double ew = pc.fac * s.e[w];
      // the segment's cubic (contours.f90:718-775), from nodes w-1 .. w+2
      long long j[4];
      j[0] = wprev(w, cs, L);
      j[1] = w;
      j[2] = wnext(w, cs, L);
      j[3] = wnext(j[2], cs, L);
      double X[4], Y[4], dx[3], dy[3], v[3], bb[2];
#pragma unroll
      for (int m = 0; m < 4; m++) {
        X[m] = in.xw[j[m]];
        Y[m] = in.yw[j[m]];
      }
#pragma unroll
      for (int m = 0; m < 3; m++) {
        const double xx = X[m + 1] - X[m];
        dx[m] = xx - c.ellx * f_dint(xx * c.hlxi);
        const double yy = Y[m + 1] - Y[m];
        dy[m] = yy - c.elly * f_dint(yy * c.hlyi);
        v[m] = dx[m] * dx[m] + dy[m] * dy[m];
      }
#pragma unroll
      for (int m = 0; m < 2; m++) {
        const double u = v[m], a = -dx[m], cc = -dy[m];
        if (dx[m + 1] * a + dy[m + 1] * cc > 0.0) {
          bb[m] = 0.0;
        } else {
          const double t1 = a * v[m + 1] - dx[m + 1] * u, t2 = cc * v[m + 1] - dy[m + 1] * u;
          bb[m] = (dx[m + 1] * cc - a * dy[m + 1]) / sqrt(t1 * t1 + t2 * t2 + c.small3);
        }
      }
      const double e1 = sqrt(v[1]);
      const double u = e1 * (bb[1] + bb[0]), cc = e1 * (bb[1] - bb[0]);
      const double A = f16 * cc - f12 * u, B = f12 * (u - cc), Cc = f13 * cc;
      long long t0 = (long long)floor(Ep) + 1, t1 = (long long)floor(Ec);
      if (t1 > n - 1) t1 = n - 1;
      if (t0 < 1) t0 = 1;
      for (long long t = t0; t <= t1; t++) {
        const double acc = Ec - (double)t;
        double pp = 1.0 - acc / ew;
        // Targets are assigned by prefix sums, whose grouping rounds: a
        // segment of density zero or at the rounding level (the zero-length
        // segments that surgery leaves where it joins two nodes) can receive
        // a target that the reference's running sum gives its neighbour, and
        // 1 - acc/ew is then far outside [0, 1] or 0/0.  Such a target is
        // placed by the prefix values that assigned it (Ep < t <= Ec, so the
        // fraction lies in (0, 1]): the segment's start, within rounding of
        // where the reference puts it.
        if (!(pp >= -1e-9 && pp <= 1.0 + 1e-9)) pp = ((double)t - Ep) / (Ec - Ep);
        const double eta = pp * (A + pp * (B + pp * Cc));
        const double xx = X[1] + pp * dx[1] - eta * dy[1];
        const double yy = Y[1] + pp * dy[1] + eta * dx[1];
        out.xo[o + t] = wrapp(xx, c.ellx, c.hlxi, c.oms);
        out.yo[o + t] = wrapp(yy, c.elly, c.hlyi, c.oms);
      }
    }
  }
}

static inline int gsz(long long work) {
  long long g = (work + 255) / 256;
  if (g < 1) g = 1;
  if (g > 148 * 16) g = 148 * 16;
  return (int)g;
}

// Steps of a density tile.
static int rn_steps(long long N) {
  // Tiles of one step while that leaves no more blocks than fit on the SMs at
  // once (a tile's steps run one after the other: 10k nodes 16 us with 1, 33
  // with 8); larger ones above, where each further tile costs its scans (1.4M
  // nodes 170, 101, 78 and 73 us with 1, 3, 8 and 16; 75k nodes 23, 24, 35 with
  // 1, 3 and 8; 1.0M nodes 86 and 91 with 8 and 16), 16 once two blocks an SM
  // are left.
  return N <= 148LL * 3 * RN_STEP       ? 1
         : N <= 148LL * 3 * RN_STEP * 4 ? 3
         : N <= 148LL * 2 * RN_STEP * 16 ? 8
         : 16;
}

RenodeWords renode_words(Arena &ar, long long N, int C) {
  const int step = rn_steps(N) * RN_STEP;
  const long long nt = (N + step - 1) / step, ct = (C + 255LL) / 256;
  RenodeWords w{};
  w.ccnt = ar.get<int>(C);
  w.nstat = ar.get<unsigned long long>(nt + ct + 2);  // then the contours' words, then the tickets
  w.job[0] = {w.ccnt, C, 0u};
  w.job[1] = {w.nstat, 2 * (nt + ct + 2), 0u};
  return w;
}

int renode_batch(casl_handle *h, Arena &ar, const RenodeIn &in, RenodeOut &out, int mode,
                 const RenodeWords *cleared) {
  cudaStream_t st = h->stream;
  const Consts &c = h->c;
  long long N = in.N;
  int C = in.C;  // capacity when in.Cdev is set
  if (C == 0 || N == 0) {
    cudaMemsetAsync(out.d_counts, 0, 3 * sizeof(int), st);
    return CASL_OK;
  }
  RenodeScratch s{};
  s.cid = in.cid ? const_cast<int *>(in.cid) : ar.get<int>(N);
  s.e = ar.get<double>(N);
  s.S = ar.get<double>(N);
  s.cc = ar.get<int>(N);
  s.cornerpos = ar.get<int>(N + 1);
  s.poff = ar.get<int>(C);
  const int rnit = rn_steps(N);
  const long long nt = (N + rnit * RN_STEP - 1) / (rnit * RN_STEP), ct = (C + 255LL) / 256;
  const RenodeWords words = cleared ? *cleared : renode_words(ar, N, C);
  s.ccnt = words.ccnt;
  s.nstat = words.nstat;
  s.cstat = s.nstat + nt;
  s.tick = reinterpret_cast<int *>(s.cstat + ct);
  s.tilev = ar.get<double>(nt);
  s.tilef = ar.get<int>(nt);
  s.err = &h->scal->error;
  // pieces: one per corner of a contour with >= 2 corners, else one per
  // contour, so at most N + C
  long long P = N + C;
  s.piece = ar.get<RnPiece>(P);
  if (ar.failed) return CASL_ENOMEM;
  if (!cleared)
    if (int rc = fill_words(st, words.job, 2)) return rc;
  int g = gsz(N);
  if (!in.cid) CASL_K(k_rn_cid, g, 256, 0, st)(in, N, s.cid);
  if (rnit == 1)
    CASL_K(k_rn_nodes<1>, (int)nt, 256, 0, st)(in, s, c);
  else if (rnit == 3)
    CASL_K(k_rn_nodes<3>, (int)nt, 256, 0, st)(in, s, c);
  else if (rnit == 8)
    CASL_K(k_rn_nodes<8>, (int)nt, 256, 0, st)(in, s, c);
  else
    CASL_K(k_rn_nodes<16>, (int)nt, 256, 0, st)(in, s, c);
  // (C may be a capacity, the count being on the device: the grid is sized
  // for the usual counts and its blocks take tiles until there are none)
  CASL_K(k_rn_contours, (int)std::min(ct, 2LL * 148), 256, 0, st)(in, s, out, c, mode);
  // four nodes a thread once that leaves every SM its blocks
  const int pu = N <= 148LL * 16 * PL_BT ? 1 : 4;
  const int gp = (int)std::min((N + pu * PL_BT - 1) / (pu * PL_BT), 148LL * 32);
  if (pu == 1)
    CASL_K(k_rn_place<1>, gp, PL_BT, 0, st)(in, s, out, c);
  else
    CASL_K(k_rn_place<4>, gp, PL_BT, 0, st)(in, s, out, c);
  return check_launch(h);
}

}  // namespace casl

// Contour surgery (contours.f90:350-683) on the GPU.
//
// The reference scans the nodes of each PV level in index order and mutates
// node positions and links as it goes, so later tests see earlier
// reconnections.  The B200 version keeps that exact semantics:
//   1. Box every segment of every level in parallel (the reference's
//      nbx = nint(1.2 sqrt(N_lev)) boxes, its bwxi/bwyi scaling); a box's
//      list is contiguous, in any order: a scan takes the lowest list index
//      that passes.
//   2. Test every node against the segments of its box in parallel on the
//      unmodified state; nodes with a passing test are marked pending.
//   3. One warp per level replays the reference loop in node order, but only
//      at pending nodes.  A reconnection marks pending every later node whose
//      tests could read what it changed: the four modified nodes, their
//      original predecessors, and every node located in a box that lists a
//      segment starting at one of those.  All other nodes would find no
//      surgery in the reference either, so the result is identical.
//   4. The new contours are the cycles of the link array, each starting at
//      its lowest node index (the reference's avail() walk); they are found
//      by pointer jumping over runs of consecutive nodes, gathered into walk
//      order and renoded in parallel (renode.cu).
#include <limits.h>
#include <math.h>
#include <stdio.h>

#include <algorithm>
#include <vector>

#include "renode.cuh"
#include "scan.cuh"
#include "state.cuh"

namespace casl {

struct LevelDesc {
  int ibeg, iend;   // node range (0-based, inclusive)
  int nbx, nby;
  int boxbase;      // first global box of the level
  int levt;         // indq value of the level
  double bwxi, bwyi;
};

// An entry of a box: x the list index (the node before the segment's first), ~x
// where only the node lies in the box (see k_sg_place); y the first node, ~y
// where it lies in this box.
struct SurgState {
  double *xq, *yq, *dx, *dy;           // mutable
  int *nextq;                          // mutable
  const double4 *g0;                   // original x, y, dx, dy of every node
  const int *nq0, *prev0, *lvl;
  const uint2 *range;                  // per box: its entries, first and end
  const int2 *ent;
  unsigned char *pending;
  // one bit per window of 512 nodes (a word per 16384) set wherever a
  // pending flag is set, so the replay skips empty windows a word at a time
  unsigned int *wsum;
  const int *err;  // set: lists may be incomplete, and nothing is tested or moved
};

__device__ __forceinline__ void set_pending(const SurgState &S, int x) {
  S.pending[x] = 1;
  atomicOr(&S.wsum[x >> 14], 1u << ((x >> 9) & 31));
}

__device__ __forceinline__ int clampi(int v, int lo, int hi) { return v < lo ? lo : (v > hi ? hi : v); }

// Box range spanned by segment (i, i+dx) (contours.f90:467-480).
__device__ __forceinline__ void seg_boxes(double x, double y, double dx, double dy, const LevelDesc &L,
                                          const Consts &c, int &mbx1, int &mbx2, int &mby1,
                                          int &mby2) {
  double dnbx = (double)L.nbx, dnby = (double)L.nby;
  if (dx > 0.0) {
    mbx1 = f_int(dnbx + L.bwxi * (x - c.xmin));
    mbx2 = f_int(dnbx + L.bwxi * (x + dx - c.xmin));
  } else {
    mbx1 = f_int(dnbx + L.bwxi * (x + dx - c.xmin));
    mbx2 = f_int(dnbx + L.bwxi * (x - c.xmin));
  }
  if (dy > 0.0) {
    mby1 = f_int(dnby + L.bwyi * (y - c.ymin));
    mby2 = f_int(dnby + L.bwyi * (y + dy - c.ymin));
  } else {
    mby1 = f_int(dnby + L.bwyi * (y + dy - c.ymin));
    mby2 = f_int(dnby + L.bwyi * (y - c.ymin));
  }
  // a wrapped segment is shorter than half the domain, so its boxes lie in
  // [nbx/2, 5/2 nbx] and it spans at most nbx/2 of them; the clamps keep nodes
  // that a failed step left out of the domain, or not finite, inside the lists
  // (the conversion of a NaN is the lowest int)
  mbx1 = clampi(mbx1, 0, 3 * L.nbx);
  mby1 = clampi(mby1, 0, 3 * L.nby);
  mbx2 = clampi(mbx2, mbx1, mbx1 + L.nbx - 1);
  mby2 = clampi(mby2, mby1, mby1 + L.nby - 1);
}

__device__ __forceinline__ int node_box(double x, double y, const LevelDesc &L, const Consts &c) {
  int bx = clampi(f_int(L.bwxi * (x - c.xmin)), 0, L.nbx - 1);
  int by = clampi(f_int(L.bwyi * (y - c.ymin)), 0, L.nby - 1);
  return L.boxbase + L.nby * bx + by;
}


// --- levels (contours.f90:374-394) and box counts (contours.f90:429-454) ----
// A new level starts where indq increases; contours arrive sorted by level.
//
// The level table: level starts, their ranks and node ranges, and endnext,
// each contour's last node linked to its first (the rest of endnext is -1 on
// entry).  A thread per contour; a block counts the starts before its own
// contours itself (coalesced reads of a few thousand words), where one block
// over all contours took 27 us for 13k of them and 158 us for 53k (an
// ensemble).  The block that finishes last sizes the boxes: nint(1.2
// sqrt(N_lev)) per side (contours.f90:403-416) and the levels' first global
// boxes.  dtot[0] = levels, dtot[1] = boxes; dtot[6] = 0 on entry.
__global__ void __launch_bounds__(SCAN_BLOCK) k_lv_all(const int *__restrict__ i1q,
                                                       const int *__restrict__ i2q,
                                                       const int *__restrict__ indq, int nq,
                                                       int npt, Consts c, LevelDesc *lev,
                                                       int *__restrict__ endnext,
                                                       int *__restrict__ dtot,
                                                       long long nbox_cap,
                                                       int *__restrict__ err) {
  CASL_PDL_ENTRY();
  __shared__ int tot, carry, last;
  const int tid = threadIdx.x, b0 = blockIdx.x * SCAN_BLOCK, j = b0 + tid;
  int before = 0;
  for (int k = tid; k < b0; k += SCAN_BLOCK) before += k == 0 || indq[k] > indq[k - 1];
  block_excl_scan<int>(before, &tot);
  before = tot;
  __syncthreads();
  int v = 0, first = 0;
  if (j < nq) {
    v = indq[j];
    const int prev = j > 0 ? indq[j - 1] : 0;
    first = j == 0 || v > prev;
    if (j > 0 && v < prev) atomicExch(err, CASL_EINVAL);
  }
  const int lv = before + block_excl_scan<int>(first, &tot) + first - 1;
  if (j < nq) {
    const int a = i1q[j], b = i2q[j];
    endnext[b] = a;  // a contour's last node links back to its first
    if (first) {
      lev[lv].ibeg = a;
      lev[lv].levt = v;
    }
    if (j == nq - 1 || indq[j + 1] > v) lev[lv].iend = b;
    if (j == nq - 1) dtot[0] = lv + 1;
  }
  __threadfence();
  __syncthreads();
  if (tid == 0) {
    last = atomicAdd(&dtot[6], 1) == (int)gridDim.x - 1;
    carry = 0;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  const int nlev = __ldcg(&dtot[0]);
  for (int base = 0; base < nlev; base += SCAN_BLOCK) {
    const int L = base + tid;
    int nb = 0;
    LevelDesc d{};
    bool ok = false;
    if (L < nlev) {
      d.ibeg = __ldcg(&lev[L].ibeg);
      d.iend = __ldcg(&lev[L].iend);
      d.levt = __ldcg(&lev[L].levt);
      if (d.ibeg < 0 || d.iend >= npt || d.iend < d.ibeg) {
        atomicExch(err, CASL_EINVAL);
      } else {
        ok = true;
        double fnq = (double)(d.iend - d.ibeg + 1);
        double fnbx = 1.2 * sqrt(fnq * c.aspect);
        double fnby = fnbx / c.aspect;
        int nbx = (int)llround(fnbx);
        nbx = max(min(nbx, c.nx), 1);
        int nby = (int)llround(fnby);
        nby = max(min(nby, c.ny), 1);
        d.nbx = nbx;
        d.nby = nby;
        d.bwxi = c.oms * (double)nbx / c.ellx;
        d.bwyi = c.oms * (double)nby / c.elly;
        nb = nbx * nby;
      }
    }
    const int ex = block_excl_scan<int>(nb, &tot) + carry;
    if (ok) {
      d.boxbase = ex;
      lev[L] = d;
    }
    __syncthreads();
    if (tid == 0) carry += tot;
    __syncthreads();
  }
  if (tid == 0) {
    dtot[1] = carry;
    if ((long long)carry > nbox_cap) atomicExch(err, CASL_ECAPACITY);
  }
}

// Every box that lists the segment (x, y, dx, dy): f(box, true); then
// f(own, false) where the first node's own box is not among them (the box a
// node is tested in and the first of its segment's are rounded apart, so a node
// on a box's edge can be in neither).  Nothing unless admit(number of boxes).
template <class A, class F>
__device__ __forceinline__ void for_boxes(double x, double y, double dx, double dy,
                                          const LevelDesc &L, const Consts &c, int own, A admit, F f) {
  int mbx1, mbx2, mby1, mby2;
  seg_boxes(x, y, dx, dy, L, c, mbx1, mbx2, mby1, mby2);
  if (!admit((mbx2 - mbx1 + 1) * (mby2 - mby1 + 1))) return;
  bool met = false;
  for (int mbx = mbx1; mbx <= mbx2; mbx++) {
    const int b0 = L.boxbase + L.nby * (mbx % L.nbx);
    for (int mby = mby1; mby <= mby2; mby++) {
      const int gb = b0 + mby % L.nby;
      met |= gb == own;
      f(gb, true);
    }
  }
  if (!met) f(own, false);
}

// work arrays dx, dy (contours.f90:397-415; dsq is dx*dx + dy*dy throughout)
// and the original state, one 32-byte record per node; the entries of every box
// are counted (bcnt, zero on entry).  Segments of more than 64 boxes are also
// added up in *far, and left out once those alone exceed the capacity: 90,000
// segments over 29,000 boxes each would take seconds to count and then be
// refused.
__global__ void k_sg_init(const double *__restrict__ xq, const double *__restrict__ yq,
                          const int *__restrict__ nextq, const int *__restrict__ endnext, int npt,
                          double *dx, double *dy, double4 *g0, int *nq0, int *prev0,
                          unsigned char *pending,
                          const LevelDesc *__restrict__ lev, const int *__restrict__ nlev_dev,
                          int *__restrict__ lvl, int *__restrict__ bcnt, long long nbox_cap,
                          unsigned long long *__restrict__ far, unsigned int ne_cap, Consts c,
                          int *err) {
  CASL_PDL_ENTRY();
  const int nlev = nlev_dev[0];
  const bool fits = nlev_dev[1] <= nbox_cap;  // (else k_lv_all has raised CASL_ECAPACITY)
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < npt; i += gridDim.x * blockDim.x) {
    // the node's level: the last level starting at or below i
    int lo = 0, hi = nlev - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (lev[mid].ibeg <= i) lo = mid; else hi = mid - 1;
    }
    lvl[i] = lo;
    int a = endnext[i] >= 0 ? endnext[i] : i + 1;
    double xi = xq[i], yi = yq[i];
    if (!(xi >= c.xmin && xi < c.xmax && yi >= c.ymin && yi < c.ymax)) atomicExch(err, CASL_EDOMAIN);
    a = clampi(a, 0, npt - 1);
    double xx = xq[a] - xi;
    double ddx = xx - c.ellx * f_dint(xx * c.hlxi);
    double yy = yq[a] - yi;
    double ddy = yy - c.elly * f_dint(yy * c.hlyi);
    dx[i] = ddx;
    dy[i] = ddy;
    double2 *g = reinterpret_cast<double2 *>(g0 + i);
    g[0] = make_double2(xi, yi);
    g[1] = make_double2(ddx, ddy);
    int nx = nextq[i];
    if (nx < 0 || nx >= npt) { atomicExch(err, CASL_EINVAL); nx = i; }
    nq0[i] = nx;
    prev0[nx] = i;
    pending[i] = 0;
    const LevelDesc L = lev[lo];
    auto admit = [&](int cnt) {
      if (!fits) return false;
      if (cnt <= 64 || atomicAdd(far, (unsigned long long)cnt) + cnt <= ne_cap) return true;
      atomicExch(err, CASL_ECAPACITY);
      return false;
    };
    for_boxes(xi, yi, ddx, ddy, L, c, node_box(xi, yi, L, c), admit,
              [&](int gb, bool) { red_add_s32(&bcnt[gb], 1); });
  }
}

__device__ __forceinline__ double4 ld_g0(const double4 *p) {
  const double2 a = reinterpret_cast<const double2 *>(p)[0], b = reinterpret_cast<const double2 *>(p)[1];
  return make_double4(a.x, a.y, b.x, b.y);
}

// The boxes' ranges in the entry array: tiles of 1024 boxes, each taking its share
// from a running total (the order of the boxes in memory is free).  The total
// is kept in 64 bits: some 80,000 segments that each span half the domain both
// ways have more than 2^31 entries.  Past the capacity (CASL_ECAPACITY is
// raised, and the kernels that read the lists return) nothing is written.
__global__ void __launch_bounds__(256) k_sg_alloc(const int *__restrict__ bcnt,
                                                  const int *__restrict__ nbox_dev,
                                                  long long nbox_cap, unsigned int ne_cap,
                                                  uint2 *__restrict__ range,
                                                  unsigned long long *__restrict__ total,
                                                  int *__restrict__ err) {
  CASL_PDL_ENTRY();
  __shared__ unsigned long long tot, base;
  const long long nbox = *nbox_dev < nbox_cap ? (long long)*nbox_dev : nbox_cap;
  for (long long t0 = blockIdx.x * 1024LL; t0 < nbox; t0 += gridDim.x * 1024LL) {
    const long long b = t0 + 4 * threadIdx.x;
    unsigned int n[4];
#pragma unroll
    for (int k = 0; k < 4; k++) n[k] = b + k < nbox ? (unsigned)bcnt[b + k] : 0u;
    unsigned long long at = block_excl_scan_any<unsigned long long>(
        (unsigned long long)n[0] + n[1] + n[2] + n[3], &tot);
    if (threadIdx.x == 0) {
      base = atomicAdd(total, tot);
      if (base + tot > ne_cap) atomicExch(err, CASL_ECAPACITY);
    }
    __syncthreads();
    at += base;
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const unsigned int st = (unsigned)(at < ne_cap ? at : ne_cap);
      if (b + k < nbox) range[b + k] = make_uint2(st, st);
      at += n[k];
    }
    __syncthreads();
  }
}

// The entries.  A box's list is contiguous so that the replay reads it 32 wide:
// as links it was built in one pass, but a warp then waits for one load per
// entry (a surgery of 40 patches of 500 nodes on one level, lists of thousands,
// 124 ms, and 23 so; isolated vortices at 1024^2, 39k nodes, 1.6 ms a step, and
// 1.1 so).  A turbulent state of 1.4M nodes: this kernel, the counts and the
// ranges take 15 us more than the links did, the candidate search 7 less, and
// the replay 3 to 50 less, as there are few or many nodes to replay.
__global__ void k_sg_place(const double4 *__restrict__ g0, const int *__restrict__ nq0,
                           const int *__restrict__ lvl, const LevelDesc *__restrict__ lev, int npt,
                           unsigned int ne_cap, uint2 *__restrict__ range, int2 *__restrict__ ent,
                           int *__restrict__ nbox_of, Consts c, int *__restrict__ err) {
  CASL_PDL_ENTRY();
  if (*reinterpret_cast<volatile int *>(err)) return;
  for (int ib = blockIdx.x * blockDim.x + threadIdx.x; ib < npt; ib += gridDim.x * blockDim.x) {
    const LevelDesc L = lev[lvl[ib]];
    const int i = nq0[ib];
    const double4 g = ld_g0(g0 + i);
    const int nb = node_box(g.x, g.y, L, c);
    nbox_of[ib] = nb;
    for_boxes(g.x, g.y, g.z, g.w, L, c, nb, [](int) { return true; }, [&](int gb, bool segment) {
      const unsigned int e = atomicAdd(&range[gb].y, 1u);
      if (e < ne_cap)
        ent[e] = make_int2(segment ? ib : ~ib, gb == nb ? ~i : i);
      else
        atomicExch(err, CASL_ECAPACITY);
    });
  }
}

// The two tests of contours.f90:542-563.
__device__ __forceinline__ bool surg_test(double xi, double yi, double xs, double ys, double dxs,
                                          double dys, double dsqs, const Consts &c) {
  double xx = xs - xi;
  double delx = xx - c.ellx * f_dint(xx * c.hlxi);
  double yy = ys - yi;
  double dely = yy - c.elly * f_dint(yy * c.hlyi);
  double aa = delx * dxs + dely * dys;
  if (aa * (aa + dsqs) + c.d4small < 0.0) {
    double cr = delx * dys - dely * dxs;
    double cc = cr * cr;
    if (cc * (cc - c.dm2 * dsqs) < 0.0) return true;
  }
  return false;
}

// Parallel candidate detection on the unmodified state.
__global__ void k_sg_candidates(SurgState S, const LevelDesc *__restrict__ lev, int npt,
                                const int *__restrict__ nbox_of, Consts c) {
  CASL_PDL_ENTRY();
  if (*S.err) return;
  for (int ib = blockIdx.x * blockDim.x + threadIdx.x; ib < npt; ib += gridDim.x * blockDim.x) {
    int i = S.nq0[ib];
    int mb = nbox_of[ib];
    const double2 xy = *reinterpret_cast<const double2 *>(S.g0 + i);
    const double xi = xy.x, yi = xy.y;
    bool hit = false;
    // two entries at a time: their loads and tests do not wait for each other
    const uint2 r = S.range[mb];
    for (unsigned int e = r.x; e < r.y && !hit; e += 2) {
      const int2 v0 = S.ent[e], v1 = e + 1 < r.y ? S.ent[e + 1] : make_int2(~0, 0);
      const int s0 = v0.x < 0 ? i : (v0.y < 0 ? ~v0.y : v0.y);
      const int s1 = v1.x < 0 ? i : (v1.y < 0 ? ~v1.y : v1.y);
      const double4 p = ld_g0(S.g0 + s0), q = ld_g0(S.g0 + s1);
      const bool t0 = surg_test(xi, yi, p.x, p.y, p.z, p.w, p.z * p.z + p.w * p.w, c);
      const bool t1 = surg_test(xi, yi, q.x, q.y, q.z, q.w, q.z * q.z + q.w * q.w, c);
      hit = (t0 && s0 != ib && s0 != i) || (t1 && s1 != ib && s1 != i);
    }
    S.pending[ib] = hit ? 1 : 0;
    if (hit) atomicOr(&S.wsum[ib >> 14], 1u << ((ib >> 9) & 31));
  }
}

__device__ __forceinline__ void mark(SurgState &S, int x, int ib, int iend) {
  if (x > ib && x <= iend) set_pending(S, x);
}

// Mark every later node whose tests may read node j's changed data.  Called
// by all 32 lanes of the level's warp with the same j: the loops over boxes
// are uniform and the entries of each box are split across the lanes.
__device__ void mark_affected(SurgState &S, const LevelDesc &L, int j, int ib, const Consts &c,
                              int lane) {
  int cand[2] = {j, S.prev0[j]};
  for (int q = 0; q < 2; q++) {
    int e = cand[q];
    if (lane == 0) mark(S, e, ib, L.iend);
    // boxes listing the segment whose list entry is e
    int i = S.nq0[e];
    int mbx1, mbx2, mby1, mby2;
    const double4 g = ld_g0(S.g0 + i);
    seg_boxes(g.x, g.y, g.z, g.w, L, c, mbx1, mbx2, mby1, mby2);
    for (int mbx = mbx1; mbx <= mbx2; mbx++) {
      int mmbx = mbx % L.nbx;
      for (int mby = mby1; mby <= mby2; mby++) {
        const uint2 r = S.range[L.boxbase + L.nby * mmbx + mby % L.nby];
        for (unsigned int k = r.x + lane; k < r.y; k += 32) {
          const int2 v = S.ent[k];
          if (v.y < 0) mark(S, v.x < 0 ? ~v.x : v.x, ib, L.iend);  // a node in this box
        }
      }
    }
  }
}

// One warp per level replays contours.f90:528-613 at pending nodes.
__global__ void k_sg_replay(SurgState S, const LevelDesc *__restrict__ lev,
                            const int *__restrict__ nlev_dev, Consts c, int *nsurg,
                            int *__restrict__ stats) {
  CASL_PDL_ENTRY();
  const int lane = threadIdx.x & 31;
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (warp >= *nlev_dev || *S.err) return;
  const LevelDesc L = lev[warp];
  // Every node, flag and box entry this warp reads or writes belongs to its
  // own level, so no other warp touches them: lane 0's updates reach the
  // other lanes through this SM's L1 after __syncwarp(), and plain cached
  // loads are coherent here.
  const unsigned char *pend = S.pending;
  double *xq = S.xq, *yq = S.yq, *dx = S.dx, *dy = S.dy;
  int *nextq = S.nextq;
  const double f12 = 0.5;
  int count = 0, npend = 0;
  long long pos = L.ibeg;
  while (pos <= L.iend) {
    int ib;
    {
      // skip the 512-node windows whose summary bit is clear (read from L2:
      // this warp's own marks arrive there by atomics)
      const long long W = pos >> 9;
      const unsigned sw = __ldcg(&S.wsum[W >> 5]) >> (W & 31);
      if (!sw) {
        pos = ((W >> 5) + 1) << 14;
        continue;
      }
      const int d = __ffs(sw) - 1;
      if (d > 0) {
        pos = (W + d) << 9;
        if (pos > L.iend) break;
      }
    }
    // Windows start at the 16-aligned position at or below pos, so the wide
    // path is taken whatever the level's first node; flags below pos (already
    // visited, or another level's) are masked out.
    const long long base = pos & ~15LL;
    if (base + 512 <= (long long)L.iend + 1) {
      // 512 flags per step: one 16-byte load per lane
      uint4 v = reinterpret_cast<const uint4 *>(pend + base)[lane];
      if (lane == 0 && pos > base) {
        const int sh = (int)(pos - base);  // 1..15 leading bytes to drop
        unsigned w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int q = 0; q < 4; q++) {
          const int drop = sh - 4 * q;  // bytes of word q below pos
          if (drop >= 4) w[q] = 0u;
          else if (drop > 0) w[q] &= ~0u << (8 * drop);
        }
        v = make_uint4(w[0], w[1], w[2], w[3]);
      }
      unsigned b = __ballot_sync(0xffffffffu, (v.x | v.y | v.z | v.w) != 0u);
      if (!b) {
        pos = base + 512;
        continue;
      }
      const int f = __ffs(b) - 1;
      int off = 0;
      if (lane == f) {
        unsigned w[4] = {v.x, v.y, v.z, v.w};
        for (int q = 0; q < 4; q++)
          if (w[q]) {
            off = 4 * q + (__ffs(w[q]) - 1) / 8;
            break;
          }
      }
      off = __shfl_sync(0xffffffffu, off, f);
      ib = (int)(base + 16 * f + off);
    } else {
      long long idx = base + lane;
      bool fl = idx >= pos && idx <= L.iend && pend[idx];
      unsigned b = __ballot_sync(0xffffffffu, fl);
      if (!b) {
        pos = base + 32;
        continue;
      }
      ib = (int)(base + __ffs(b) - 1);
    }
    __syncwarp();
    npend++;
    int i = nextq[ib];
    double xi = xq[i], yi = yq[i];
    int mb = node_box(xi, yi, L, c);
    const uint2 list = S.range[mb];
    // The reference walks the box's segments in list order and continues
    // after each reconnection with the moved node.  The box list is stored
    // unordered, so each round takes the passing segment with the smallest
    // list index above the last one taken.
    int thr = -1;
    while (true) {
      int best = INT_MAX;
      for (unsigned int k = list.x + lane; k < list.y; k += 32) {
        const int isb = S.ent[k].x;
        if (isb > thr && isb < best) {
          const int is = nextq[isb];
          if (!(is == ib || is == i)) {
            const double ex = dx[is], ey = dy[is];
            if (surg_test(xi, yi, xq[is], yq[is], ex, ey, ex * ex + ey * ey, c)) best = isb;
          }
        }
      }
      for (int o = 16; o > 0; o >>= 1) best = min(best, __shfl_xor_sync(0xffffffffu, best, o));
      if (best == INT_MAX) break;
      int inew = 0, tsb = 0;
      if (lane == 0) {
        int isb = best;
        int is = nextq[isb];
        double xx = xq[is] - xq[i];
        double delx = xx - c.ellx * f_dint(xx * c.hlxi);
        double yy = yq[is] - yq[i];
        double dely = yy - c.elly * f_dint(yy * c.hlyi);
        double aa = delx * dx[is] + dely * dy[is];
        double dxa, dya;
        if (dx[is] * dx[is] + dy[is] * dy[is] + 2.0 * aa < 0.0) {
          dxa = f12 * (delx + dx[is]);
          dya = f12 * (dely + dy[is]);
          isb = is;
          is = nextq[is];
        } else {
          dxa = f12 * delx;
          dya = f12 * dely;
        }
        xx = xq[i] + dxa;
        xq[i] = wrapp(xx, c.ellx, c.hlxi, c.oms);
        yy = yq[i] + dya;
        yq[i] = wrapp(yy, c.elly, c.hlyi, c.oms);
        dx[i] = dx[i] - dxa;
        dy[i] = dy[i] - dya;
        nextq[isb] = i;
        dx[isb] = dx[isb] - dxa;
        dy[isb] = dy[isb] - dya;
        xq[is] = xq[i];
        yq[is] = yq[i];
        dx[is] = dx[is] + dxa;
        dy[is] = dy[is] + dya;
        nextq[ib] = is;
        dx[ib] = dx[ib] + dxa;
        dy[ib] = dy[ib] + dya;
        tsb = isb;
        inew = is;
        count++;
      }
      __syncwarp();  // lane 0's moves are visible to the whole warp
      const int is_new = __shfl_sync(0xffffffffu, inew, 0);
      const int isb_new = __shfl_sync(0xffffffffu, tsb, 0);
      {
        const int touched[4] = {i, is_new, isb_new, ib};
        for (int q = 0; q < 4; q++) mark_affected(S, L, touched[q], ib, c, lane);
      }
      __syncwarp();  // marks visible before the next flag scan
      i = is_new;
      xi = xq[i];
      yi = yq[i];
      if (i == ib) break;
      thr = best;
    }
    pos = ib + 1;
  }
  if (lane == 0 && count) atomicAdd(nsurg, count);
  if (stats && lane == 0) {  // trace only: pending nodes visited, surgeries
    stats[2 * warp] = npend;
    stats[2 * warp + 1] = count;
  }
}

// ---------------------------------------------------------------------------
// Rebuild: cycles of nextq -> walk-ordered contours (contours.f90:621-663)
// ---------------------------------------------------------------------------
// Runs of consecutive links, numbered in node order: tiles of 2048 nodes, each
// counting its runs and looking back for those before it.  rid: the run of
// every node; rs, re: a run's first and last node; *R their number.
constexpr int RB_TILE = 2048;
__global__ void __launch_bounds__(256) k_rb_runs(const int *__restrict__ nextq, int npt,
                                                 int *__restrict__ tick,
                                                 unsigned long long *__restrict__ stat,
                                                 int *__restrict__ rid, int *__restrict__ rs,
                                                 int *__restrict__ re, int *__restrict__ R,
                                                 int *__restrict__ err) {
  CASL_PDL_ENTRY();
  __shared__ int tot, before;
  const int tile = lb_ticket(tick);
  const int i0 = tile * RB_TILE + 8 * (int)threadIdx.x;  // 8 consecutive nodes
  unsigned st = 0, en = 0;
  if (i0 < npt) {
    int prev = i0 > 0 ? nextq[i0 - 1] : -1;
#pragma unroll
    for (int k = 0; k < 8; k++)
      if (i0 + k < npt) {
        const int nx = nextq[i0 + k];
        st |= (unsigned)(i0 + k == 0 || prev != i0 + k) << k;
        en |= (unsigned)(nx != i0 + k + 1) << k;
        prev = nx;
      }
  }
  int r = block_excl_scan_any<int>(__popc(st), &tot);
  if (threadIdx.x < 32) {
    const unsigned long long pre = lb_prefix(stat, tile, (unsigned)tot, err);
    if (threadIdx.x == 0) before = (int)pre;
  }
  __syncthreads();
  r += before - 1;
#pragma unroll
  for (int k = 0; k < 8; k++)
    if (i0 + k < npt) {
      if (st >> k & 1) rs[++r] = i0 + k;
      rid[i0 + k] = r;
      if (en >> k & 1) re[r] = i0 + k;
    }
  if ((tile + 1) * (long long)RB_TILE >= npt && threadIdx.x == 0) *R = before + tot;
}

// Every run: its successor run; a run that closes on itself is a whole
// contour (head, length); the others (the few runs surgery cut and joined)
// go to the multi list for k_rb_cycles_block.  Grid-wide.
__global__ void k_rb_cycles_pre(const int *__restrict__ nextq, const int *__restrict__ rid,
                                const int *__restrict__ rs, const int *__restrict__ re,
                                const int *__restrict__ R_dev, int *__restrict__ nr,
                                int *__restrict__ lab, int *__restrict__ nrj,
                                int *__restrict__ hr, int *__restrict__ val,
                                int *__restrict__ ishead, int *__restrict__ multi, int *__restrict__ nmulti) {
  CASL_PDL_ENTRY();
  const int R = *R_dev;
  for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < R; r += gridDim.x * blockDim.x) {
    const int t = rid[nextq[re[r]]];
    nr[r] = t;
    const int len = re[r] - rs[r] + 1;
    lab[r] = rs[r];
    if (t == r) {  // a whole contour
      hr[r] = r;
      ishead[r] = 1;
      val[r] = len;
    } else {
      nrj[r] = t;
      multi[atomicAdd(nmulti, 1)] = r;
    }
  }
}

// The cycles through the multi-run list: one block, pointer jumping over
// the M runs in shared order.
__global__ void __launch_bounds__(1024) k_rb_cycles_block(
    const int *__restrict__ nextq, const int *__restrict__ rid, const int *__restrict__ rs,
    const int *__restrict__ re, const int *__restrict__ R_dev, int *__restrict__ nr,
    int *lab, int *lab2, int *nrj, int *nrj2, int *__restrict__ hr, int *succ, int *succ2,
    int *val, int *val2, int *__restrict__ ishead, int *__restrict__ multi,
    const int *__restrict__ nmulti) {
  CASL_PDL_ENTRY();
  const int M = *nmulti;
  int rounds = 1;
  while ((1 << rounds) < M) rounds++;
  rounds++;
  for (int it = 0; it < rounds && M > 0; it++) {
    for (int q = threadIdx.x; q < M; q += blockDim.x) {
      int r = multi[q];
      int n = nrj[r];
      lab2[r] = min(lab[r], lab[n]);
      nrj2[r] = nrj[n];
    }
    __syncthreads();
    for (int q = threadIdx.x; q < M; q += blockDim.x) {
      int r = multi[q];
      lab[r] = lab2[r];
      nrj[r] = nrj2[r];
    }
    __syncthreads();
  }
  for (int q = threadIdx.x; q < M; q += blockDim.x) {
    int r = multi[q];
    int h = rid[lab[r]];
    hr[r] = h;
    succ[r] = nr[r] == h ? -1 : nr[r];
    val[r] = re[r] - rs[r] + 1;
    ishead[r] = h == r;
  }
  __syncthreads();
  for (int it = 0; it < rounds && M > 0; it++) {
    for (int q = threadIdx.x; q < M; q += blockDim.x) {
      int r = multi[q];
      int sc = succ[r];
      val2[r] = val[r] + (sc >= 0 ? val[sc] : 0);
      succ2[r] = sc >= 0 ? succ[sc] : -1;
    }
    __syncthreads();
    for (int q = threadIdx.x; q < M; q += blockDim.x) {
      int r = multi[q];
      val[r] = val2[r];
      succ[r] = succ2[r];
    }
    __syncthreads();
  }
}

// The contours: the head runs in order, their first walk positions, lengths and
// levels.  Tiles of 256 runs, scanned by looking back (contours * 2^31 +
// nodes); cidx is written for head runs only.  *C the number of contours.
__global__ void __launch_bounds__(256) k_rb_contours(const int *__restrict__ ishead,
                                                     const int *__restrict__ val,
                                                     const int *__restrict__ rs,
                                                     const int *__restrict__ lvl,
                                                     const LevelDesc *__restrict__ lev,
                                                     const int *__restrict__ R_dev,
                                                     int *__restrict__ tick,
                                                     unsigned long long *__restrict__ stat,
                                                     int *__restrict__ cidx, int *__restrict__ cst,
                                                     int *__restrict__ clen, int *__restrict__ clev,
                                                     int *__restrict__ C, int *__restrict__ err) {
  CASL_PDL_ENTRY();
  __shared__ unsigned long long tot, before;
  const int R = *R_dev, ntile = (R + 255) / 256;
  while (true) {
    const int tile = lb_ticket(tick);
    if (tile >= ntile) return;
    const int r = tile * 256 + threadIdx.x;
    const bool f = r < R && ishead[r];
    const int len = f ? val[r] : 0;
    unsigned long long at =
        block_excl_scan_any<unsigned long long>(f ? (1ull << 31) + (unsigned)len : 0ull, &tot);
    if (threadIdx.x < 32) {
      const unsigned long long pre = lb_prefix(stat, tile, tot, err);
      if (threadIdx.x == 0) before = pre;
    }
    __syncthreads();
    at += before;
    if (f) {
      const int c = (int)(at >> 31);
      cidx[r] = c;
      cst[c] = (int)(at & 0x7fffffffull);
      clen[c] = len;
      clev[c] = lev[lvl[rs[r]]].levt;
    }
    if (tile == ntile - 1 && threadIdx.x == 0) *C = (int)((before + tot) >> 31);
  }
}

__global__ void k_rb_gather2(const double *__restrict__ xq, const double *__restrict__ yq, int npt,
                             const int *__restrict__ rid, const int *__restrict__ rs,
                             const int *__restrict__ hr, const int *__restrict__ cidx,
                             const int *__restrict__ val, const int *__restrict__ cst,
                             const int *__restrict__ clen, double *__restrict__ xw,
                             double *__restrict__ yw, int *__restrict__ cidw) {
  CASL_PDL_ENTRY();
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < npt; i += gridDim.x * blockDim.x) {
    const int r = rid[i];
    const int c = cidx[hr[r]];
    const int pos = cst[c] + (clen[c] - val[r]) + (i - rs[r]);
    xw[pos] = xq[i];
    yw[pos] = yq[i];
    cidw[pos] = c;
  }
}

// Write the renoded contours back into the node and contour arrays
// (contours.f90:645-680) using the counts left in device memory.
__global__ void k_rb_writeback(const int *__restrict__ cnt, long long npm, long long nm,
                               const int *__restrict__ ocs, const int *__restrict__ olen,
                               const int *__restrict__ olev, const double *__restrict__ xo,
                               const double *__restrict__ yo, double *__restrict__ xq,
                               double *__restrict__ yq, int *__restrict__ nextq,
                               int *__restrict__ i1q, int *__restrict__ i2q,
                               int *__restrict__ npq, int *__restrict__ indq,
                               Scalars *__restrict__ s, int M, double twist) {
  CASL_PDL_ENTRY();
  const int nq = cnt[0], npt = cnt[1];
  if (blockIdx.x == 0)  // (a launch of its own took 2 us of a step)
    for (int m = threadIdx.x; m < M; m += blockDim.x) s[m].twist = s[m].twist - twist;
  if (cnt[2] || npt > npm || nq > nm) {
    if (blockIdx.x == 0 && threadIdx.x == 0) atomicExch(&s->error, CASL_ECAPACITY);
    return;
  }
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < nq; j += gridDim.x * blockDim.x) {
    i1q[j] = ocs[j];
    i2q[j] = ocs[j] + olen[j] - 1;
    npq[j] = olen[j];
    indq[j] = olev[j];
  }
  for (long long b = blockIdx.x * (long long)CC_CHUNK; b < npt; b += (long long)gridDim.x * CC_CHUNK) {
    chunk_contours(ocs, nq, b);
    for (int i = (int)b + threadIdx.x; i < min((long long)npt, b + CC_CHUNK); i += blockDim.x) {
      xq[i] = xo[i];
      yq[i] = yo[i];
      const int j = chunk_contour_of(ocs, nq, i);
      nextq[i] = i + 1 < ocs[j] + olen[j] ? i + 1 : ocs[j];
    }
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    s->nq = nq;
    s->nptq = npt;
  }
}

__global__ void k_twist_sub(Scalars *s, int M, double twist) {
  CASL_PDL_ENTRY();
  for (int m = threadIdx.x; m < M; m += blockDim.x) s[m].twist = s[m].twist - twist;
}

static inline int gs(long long work) {
  long long g = (work + 255) / 256;
  if (g < 1) g = 1;
  if (g > 148 * 16) g = 148 * 16;
  return (int)g;
}

// Walk-ordered contours of the current link array + renode + write back.
// Issues no host synchronisation: every count stays in device memory and
// every buffer is sized from the node count npt.  stat (see surgery_dev) and
// rw's words are zero.
static int rebuild_and_renode(casl_handle *h, Arena &ar, int npt, const int *lvl,
                              const LevelDesc *dlev, unsigned long long *stat,
                              const RenodeWords &rw, double twist) {
  cudaStream_t st = h->stream;
  int *rid = ar.get<int>(npt);
  int *dtot = ar.get<int>(8);
  // run arrays (R <= npt)
  int *rs = ar.get<int>(npt), *re = ar.get<int>(npt), *nr = ar.get<int>(npt);
  int *lab = ar.get<int>(npt), *lab2 = ar.get<int>(npt), *nrj = ar.get<int>(npt);
  int *nrj2 = ar.get<int>(npt), *hr = ar.get<int>(npt), *succ = ar.get<int>(npt);
  int *succ2 = ar.get<int>(npt), *ishead = ar.get<int>(npt), *cidx = ar.get<int>(npt);
  int *val = ar.get<int>(npt), *val2 = ar.get<int>(npt);
  int *multi = ar.get<int>(npt);
  // cycles (C <= R <= npt)
  int *clen = ar.get<int>(npt), *clev = ar.get<int>(npt), *cst = ar.get<int>(npt);
  double *xw = ar.get<double>(npt), *yw = ar.get<double>(npt);
  int *ocs = ar.get<int>(npt), *olen = ar.get<int>(npt), *olev = ar.get<int>(npt);
  int *cnt = ar.get<int>(4);
  int *cidw = ar.get<int>(npt);
  const int rt = (npt + RB_TILE - 1) / RB_TILE, ct = (npt + 255) / 256;
  if (ar.failed) return CASL_ENOMEM;
  int *tick = reinterpret_cast<int *>(stat + rt + ct), *nmulti = tick + 2, *err = &h->scal->error;
  const int g = gs(npt);
  CASL_K(k_rb_runs, rt, 256, 0, st)(h->nextq, npt, tick, stat, rid, rs, re, dtot, err);  // dtot[0] = R
  CASL_K(k_rb_cycles_pre, g, 256, 0, st)(h->nextq, rid, rs, re, dtot, nr, lab, nrj, hr, val, ishead,
                                         multi, nmulti);
  CASL_K(k_rb_cycles_block, 1, 1024, 0, st)(h->nextq, rid, rs, re, dtot, nr, lab, lab2, nrj, nrj2,
                                            hr, succ, succ2, val, val2, ishead, multi, nmulti);
  // (the run count is on the device: blocks take tiles until there are none)
  CASL_K(k_rb_contours, std::min(ct, 2 * 148), 256, 0, st)(ishead, val, rs, lvl, dlev, dtot, tick + 1,
                                                           stat + rt, cidx, cst, clen, clev,
                                                           dtot + 1, err);  // dtot[1] = C
  CASL_K(k_rb_gather2, g, 256, 0, st)(h->xq, h->yq, npt, rid, rs, hr, cidx, val, cst, clen, xw, yw,
                                      cidw);
  int rc = check_launch(h);
  if (rc) return rc;
  RenodeIn in{xw, yw, cst, clen, clev, npt, npt, dtot + 1, cidw};
  RenodeOut out{};
  out.xo = h->xqi;  // node-sized scratch of the RK step, free between steps
  out.yo = h->yqi;
  out.ocs = ocs; out.olen = olen; out.olev = olev;
  out.cap = h->npm;
  out.d_counts = cnt;
  rc = renode_batch(h, ar, in, out, RENODE_SURGERY, &rw);
  if (rc) return rc;
  CASL_K(k_rb_writeback, gs(h->npm < (1 << 24) ? h->npm : (1 << 24)), 256, 0, st)(
      cnt, h->npm, h->nm, ocs, olen, olev, h->xqi, h->yqi, h->xq, h->yq, h->nextq, h->i1q,
      h->i2q, h->npq, h->indq, h->scal, h->M, twist);
  return check_launch(h);
}

int surgery_dev(casl_handle *h, double twist) {
  cudaStream_t st = h->stream;
  if (h->nq == 0 || h->nptq == 0) {
    if (twist != 0.0) CASL_K(k_twist_sub, 1, 256, 0, st)(h->scal, h->M, twist);
    return check_launch(h);
  }
  const Consts &c = h->c;
  const int nq = h->nq, npt = h->nptq;
  const long long nbox_cap = 2LL * npt + nq + 64;
  const unsigned int ne_cap = (unsigned)std::min(20LL * npt + 64, (long long)INT_MAX);
  // (305 bytes a node beside the boxes and their entries)
  size_t need = (size_t)npt * 400 + (size_t)nq * 96 + (size_t)nbox_cap * 12 +
                (size_t)ne_cap * 8 + ((size_t)64 << 20);
  int rc = ensure_scratch(h, need);
  if (rc) return rc;
  Arena ar{(char *)h->sx, h->sx_bytes, 0};
  int *err = &h->scal->error;
  Trace tr;
  tr.begin(st, "start");
  // levels and boxes, on the device
  LevelDesc *dlev = ar.get<LevelDesc>(nq);
  // [0] nlev, [1] nbox, [2..3] entries (64 bits), [4] nsurg, [6] blocks done,
  // [8..9] entries of segments over many boxes (64 bits)
  int *dtot = ar.get<int>(16);
  int *endnext = ar.get<int>(npt), *lvl = ar.get<int>(npt);
  double *dx = ar.get<double>(npt), *dy = ar.get<double>(npt);
  double4 *g0 = ar.get<double4>(npt);
  int *nq0 = ar.get<int>(npt), *prev0 = ar.get<int>(npt);
  unsigned char *pending = ar.get<unsigned char>(npt + 16);
  unsigned int *wsum = ar.get<unsigned int>((npt >> 14) + 2);
  int *nbox_of = ar.get<int>(npt), *bcnt = ar.get<int>(nbox_cap);
  uint2 *range = ar.get<uint2>(nbox_cap);
  int2 *ent = ar.get<int2>(ne_cap);
  // status words of the rebuild's run and contour tiles, then their tickets and
  // the number of cut runs; and the renode's words
  const long long nstat = (npt + RB_TILE - 1) / RB_TILE + (npt + 255) / 256 + 2;
  unsigned long long *stat = ar.get<unsigned long long>(nstat);
  const RenodeWords rw = renode_words(ar, npt, npt);
  if (ar.failed) return CASL_ENOMEM;
  const int g = gs(npt);
  {
    // everything the whole surgery needs cleared, in one launch
    const FillJob z[7] = {{endnext, npt, 0xffffffffu},
                          {bcnt, nbox_cap, 0u},
                          {wsum, (npt >> 14) + 2, 0u},
                          {dtot + 2, 8, 0u},
                          {stat, 2 * nstat, 0u},
                          rw.job[0],
                          rw.job[1]};
    if (int rc = fill_words(st, z, 7)) return rc;
  }
  CASL_K(k_lv_all, (nq + SCAN_BLOCK - 1) / SCAN_BLOCK, SCAN_BLOCK, 0, st)(
      h->i1q, h->i2q, h->indq, nq, npt, c, dlev, endnext, dtot, nbox_cap, err);
  CASL_K(k_sg_init, g, 256, 0, st)(h->xq, h->yq, h->nextq, endnext, npt, dx, dy, g0, nq0, prev0,
                                   pending, dlev, dtot, lvl, bcnt, nbox_cap,
                                   reinterpret_cast<unsigned long long *>(dtot + 8), ne_cap, c, err);
  CASL_K(k_sg_alloc, (int)std::min((nbox_cap + 1023) / 1024, 148LL * 8), 256, 0, st)(
      bcnt, dtot + 1, nbox_cap, ne_cap, range, reinterpret_cast<unsigned long long *>(dtot + 2), err);
  CASL_K(k_sg_place, g, 256, 0, st)(g0, nq0, lvl, dlev, npt, ne_cap, range, ent, nbox_of, c, err);
  SurgState S{};
  S.xq = h->xq; S.yq = h->yq; S.dx = dx; S.dy = dy; S.nextq = h->nextq;
  S.g0 = g0; S.nq0 = nq0; S.prev0 = prev0; S.lvl = lvl;
  S.range = range; S.ent = ent;
  S.pending = pending;
  S.wsum = wsum;
  S.err = err;
  tr.point("binning");
  CASL_K(k_sg_candidates, g, 256, 0, st)(S, dlev, npt, nbox_of, c);
  tr.point("candidates");
  int *stats = tr.on ? ar.get<int>(2 * (size_t)nq) : nullptr;
  if (stats) CASL_CUDA_TRY(cudaMemsetAsync(stats, 0, 2 * (size_t)nq * sizeof(int), st));
  CASL_K(k_sg_replay, (nq * 32 + 127) / 128, 128, 0, st)(S, dlev, dtot + 0, c, dtot + 4, stats);
  rc = check_launch(h);
  if (rc) return rc;
  tr.point("replay");
  if (stats) {
    std::vector<int> hs(2 * (size_t)nq);
    int nlev = 0;
    CASL_CUDA_TRY(cudaMemcpyAsync(hs.data(), stats, hs.size() * sizeof(int), cudaMemcpyDeviceToHost, st));
    CASL_CUDA_TRY(cudaMemcpyAsync(&nlev, dtot, sizeof(int), cudaMemcpyDeviceToHost, st));
    CASL_CUDA_TRY(cudaStreamSynchronize(st));
    long long sp = 0, ss = 0;
    int mp = 0, ms = 0, wl = 0;
    for (int l = 0; l < nlev; l++) {
      sp += hs[2 * l];
      ss += hs[2 * l + 1];
      if (hs[2 * l] > mp) { mp = hs[2 * l]; wl = l; }
      ms = std::max(ms, hs[2 * l + 1]);
    }
    fprintf(stderr, "[casl trace] replay: %d levels, pending %lld (max %d at level %d, %d surgeries there), surgeries %lld (max %d)\n",
            nlev, sp, mp, wl, hs[2 * wl + 1], ss, ms);
  }
  rc = rebuild_and_renode(h, ar, npt, lvl, dlev, stat, rw, twist);
  if (rc) return rc;
  tr.point("rebuild+renode");
  tr.flush("surgery");
  // the host copies of the counts are refreshed at the next synchronisation
  return CASL_OK;
}

// Renode of one contour supplied by the host (casl_renode).
int renode_host(casl_handle *h, const double *xd, const double *yd, int npd, double *xr,
                double *yr, int cap, int *npr) {
  cudaStream_t st = h->stream;
  size_t need = (size_t)npd * 200 + (size_t)cap * 16 + ((size_t)16 << 20);
  int rc = ensure_scratch(h, need);
  if (rc) return rc;
  Arena ar{(char *)h->sx, h->sx_bytes, 0};
  double *xw = ar.get<double>(npd), *yw = ar.get<double>(npd);
  double *xo = ar.get<double>(cap + 1), *yo = ar.get<double>(cap + 1);
  int *cs = ar.get<int>(1), *len = ar.get<int>(1);
  RenodeOut out{};
  out.xo = xo; out.yo = yo;
  out.ocs = ar.get<int>(1); out.olen = ar.get<int>(1); out.olev = ar.get<int>(1);
  out.cap = cap;
  out.d_counts = ar.get<int>(4);
  if (ar.failed) return CASL_ENOMEM;
  int z = 0;
  CASL_CUDA_TRY(cudaMemcpyAsync(xw, xd, npd * sizeof(double), cudaMemcpyHostToDevice, st));
  CASL_CUDA_TRY(cudaMemcpyAsync(yw, yd, npd * sizeof(double), cudaMemcpyHostToDevice, st));
  CASL_CUDA_TRY(cudaMemcpyAsync(cs, &z, sizeof(int), cudaMemcpyHostToDevice, st));
  CASL_CUDA_TRY(cudaMemcpyAsync(len, &npd, sizeof(int), cudaMemcpyHostToDevice, st));
  RenodeIn in{xw, yw, cs, len, nullptr, 1, npd};
  rc = renode_batch(h, ar, in, out, RENODE_PLAIN);
  if (rc) return rc;
  int hc[3];
  CASL_CUDA_TRY(cudaMemcpyAsync(hc, out.d_counts, 3 * sizeof(int), cudaMemcpyDeviceToHost, st));
  CASL_CUDA_TRY(cudaStreamSynchronize(st));
  if (hc[2]) return CASL_ECAPACITY;
  *npr = hc[1];
  if (hc[1] > 0) {
    CASL_CUDA_TRY(cudaMemcpyAsync(xr, xo, hc[1] * sizeof(double), cudaMemcpyDeviceToHost, st));
    CASL_CUDA_TRY(cudaMemcpyAsync(yr, yo, hc[1] * sizeof(double), cudaMemcpyDeviceToHost, st));
    CASL_CUDA_TRY(cudaStreamSynchronize(st));
  }
  return check_launch(h);
}

}  // namespace casl

// Parallel node redistribution of many closed contours at once
// (renode, contours.f90:687-933).
//
// Input: contours stored contiguously in "walk order" (node k of contour c at
// cs[c] + k, the reference's xd(k+1)).  Every step of the reference's renode
// is a stencil over a node and its cyclic neighbours, so it runs one thread
// per node; the sequential "acc" walk that places new nodes becomes a
// segmented prefix sum of the node densities e(i) per contour, each old
// segment then emitting the new nodes whose cumulative density falls in it.
// Corners split a contour into pieces exactly as the reference's ncorn >= 2
// branch does.  Node counts (nint of the density sums) and the placement
// formula are the reference's; only the summation order of e(i) differs.
#pragma once

#include "common.cuh"
#include "scan.cuh"

namespace casl {

enum RenodeMode { RENODE_SURGERY = 0, RENODE_PLAIN = 1 };

struct RenodeIn {
  const double *xw, *yw;  // walk layout, N nodes
  const int *cs, *len;    // per contour
  const int *levt;        // per contour level index (copied to the output)
  int C;                  // contours (an upper bound when Cdev is given)
  long long N;            // nodes
  const int *Cdev;        // optional: the contour count in device memory
  const int *cid;         // optional: the contour of every walk node (else searched)
};

__device__ __forceinline__ int contours_in(const RenodeIn &in) { return in.Cdev ? *in.Cdev : in.C; }

struct RenodeOut {
  double *xo, *yo;        // output nodes (capacity cap)
  int *ocs, *olen, *olev; // output contours (capacity C)
  long long cap;
  int *d_counts;          // [0] contours kept, [1] nodes, [2] overflow flag
};

__device__ __forceinline__ int contour_of(const int *__restrict__ cs, int C, long long w) {
  int lo = 0, hi = C - 1;
  while (lo < hi) {
    int mid = (lo + hi + 1) >> 1;
    if (cs[mid] <= w) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// The contour of every node of a chunk of CC_CHUNK nodes (a block's): one search
// in memory for the first, the following starts staged in shared memory and
// searched there (beyond them, in memory again).
constexpr int CC_CHUNK = 1024, CC_STARTS = 256;
struct ChunkContours {
  int j0, st[CC_STARTS];
};
__device__ __forceinline__ ChunkContours &chunk_shared() {
  __shared__ ChunkContours c;
  return c;
}
__device__ __forceinline__ void chunk_contours(const int *__restrict__ cs, int C, long long w0) {
  ChunkContours &c = chunk_shared();
  __syncthreads();
  if (threadIdx.x < 32) {  // 32-way search: the last contour starting at or before w0
    int lo = 0, hi = C;    // cs[lo] <= w0, and w0 < cs[hi] (hi = C: none)
    while (hi - lo > 1) {
      const int step = (hi - lo + 31) / 32, at = lo + step * (int)threadIdx.x;
      const unsigned m = __ballot_sync(0xffffffffu, at < hi && cs[at] <= w0);
      const int last = 31 - __clz(m | 1u);
      hi = min(hi, lo + step * (last + 1));
      lo = lo + step * last;
    }
    if (threadIdx.x == 0) c.j0 = lo;
  }
  __syncthreads();
  for (int t = threadIdx.x; t < CC_STARTS; t += blockDim.x)
    c.st[t] = c.j0 + t < C ? cs[c.j0 + t] : 0x7fffffff;
  __syncthreads();
}
__device__ __forceinline__ int chunk_contour_of(const int *__restrict__ cs, int C, long long w) {
  const ChunkContours &c = chunk_shared();
  if (c.st[CC_STARTS - 1] <= w) return contour_of(cs, C, w);
  int lo = 0, hi = CC_STARTS - 1;  // st[lo] <= w < st[hi]
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (c.st[mid] <= w) lo = mid; else hi = mid;
  }
  return c.j0 + lo;
}

// A piece of a contour between corners (or all of it): first node, nodes, new
// nodes, where those go; new nodes per density; the contour's prefix sum before
// the first node, and the rest of its total.
struct __align__(16) RnPiece {
  int st, len, n, out;
  double fac, preA, preW, pad;
};
struct RenodeScratch {
  int *cid;                  // contour of each walk node
  double *e, *S;              // node densities, and their sums along the contour
  int *cc;                   // 2 * (corners before the node) + (the node is one)
  int *ccnt;                 // corners per contour
  int *poff;                 // per contour: its first piece (-1: the contour is not kept)
  RnPiece *piece;
  int *cornerpos;
  // tiles of the two scans: tickets, status words, and the node tiles'
  // densities since their last contour start
  int *tick;                 // [0] nodes, [1] contours, [2] pieces allotted
  unsigned long long *nstat, *cstat;
  double *tilev;
  int *tilef;
  int *err;
};

// Renodes every contour; issues no host synchronisation.  out.d_counts
// receives [kept contours, kept nodes, overflow flag]; on overflow (kept
// nodes > out.cap) nothing is written to the output arrays and the caller
// reports CASL_ECAPACITY when it reads the counts.
// The words a renode needs at zero (corner counts, tile words and tickets) are
// cleared by renode_batch itself, or by a caller that clears other words
// anyway: it allocates them (from the same arena, for the same N and C), clears
// them with its own, and hands them over.
struct RenodeWords {
  int *ccnt;
  unsigned long long *nstat;
  FillJob job[2];
};
RenodeWords renode_words(Arena &ar, long long N, int C);
int renode_batch(casl_handle *h, Arena &ar, const RenodeIn &in, RenodeOut &out, int mode,
                 const RenodeWords *cleared = nullptr);

}  // namespace casl

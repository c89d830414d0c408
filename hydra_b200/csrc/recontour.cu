// Recontouring (congen.f90:24-441) on the GPU.
//
// 1. Ultra-fine field (16x): contour PV from integer jump counts
//    (con2ugrid, congen.f90:338-441) plus the bilinear residual
//    (congen.f90:45-61), or the bilinear field alone when there are no
//    contours (congen.f90:63-95).
// 2. Crossings are numbered by edge in the reference's order (x lines: ix outer
//    / iy inner, then y lines: iy outer / ix inner, congen.f90:200-254), from
//    per-edge counts, and contours are followed box by box inside tiles of
//    the grid (trace.cuh); the pieces are linked and ranked.
// 3. Only boxes with two out-crossings of a level (saddles) depend on the
//    order of the reference's traversal, so those few are resolved by a short
//    exact simulation of that traversal over the lists between them.
// 4. Each contour starts at its lowest-numbered crossing (the reference's
//    `free` loop); contours are ordered by level then by that crossing,
//    gathered into walk order and renoded three times (congen.f90:295-310).
// With beta != 0 the PV is not periodic in y and recontouring follows
// econgen.f90 (the reference's ecaps build) instead: the level range and the
// rows iymin..iymax that it needs come from the field's row extremes, the
// rows outside the basic box are its periodic images offset by beta*Ly per
// box, crossings are enumerated over that extended grid in econgen's order,
// and of the traced contours only one periodic image each is kept, its y
// folded back into the box, before the renodes.
#include <cub/device/device_radix_sort.cuh>
#include <math.h>
#include <stdio.h>
#include <stdlib.h>

#include <algorithm>
#include <atomic>
#include <vector>

#include "renode.cuh"
#include "scan.cuh"
#include "state.cuh"

namespace casl {

// ---------------------------------------------------------------------------
// Ultra-fine field
// ---------------------------------------------------------------------------
__global__ void k_u_scatter(const double *__restrict__ xq, const double *__restrict__ yq,
                            const int *__restrict__ nextq, int npt, double qjump,
                            int *__restrict__ J, int *__restrict__ ljx, Consts c,
                            int *__restrict__ err) {
  CASL_PDL_ENTRY();
  const int nxu = c.nxu, nyu = c.nyu;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < npt; i += gridDim.x * blockDim.x) {
    int ia = nextq[i];
    if (ia < 0 || ia >= npt) { atomicExch(err, CASL_EINVAL); continue; }
    double xi = xq[i], yi = yq[i], xa = xq[ia], ya = yq[ia];
    if (!(xi >= c.xmin && xi < c.xmax && yi >= c.ymin && yi < c.ymax)) {
      atomicExch(err, CASL_EDOMAIN);
      continue;
    }
    int ixci = f_int(c.glxui * (xi - c.xmin));
    int ixca = f_int(c.glxui * (xa - c.xmin));
    double xx = xa - xi;
    double dx = xx - c.ellx * f_dint(xx * c.hlxi);
    double yy = ya - yi;
    double dy = yy - c.elly * f_dint(yy * c.hlyi);
    int ixdif = ixca - ixci;
    int nxc = ixdif - nxu * ((2 * ixdif) / nxu);
    if (fabs(yy) > c.hly) {
      double cc = f_sign1(dy);
      double p = -(yi - c.hly * cc) / (dy + c.small);
      int ix = 1 + f_int(c.glxui * fmod(c.ellx + c.hlx + xi + p * dx, c.ellx));
      ix = ix < 1 ? 1 : (ix > nxu ? nxu : ix);
      red_add_s32(&ljx[ix - 1], -(int)cc);
    }
    if (nxc != 0 && nxc >= -nxu && nxc <= nxu) {
      int jump = f_isign1(nxc);
      int ixbeg = ixci + (1 + jump) / 2 + nxu;
      for (int ncr = 0; ncr != nxc; ncr += jump) {
        int m = (ixbeg + ncr) % nxu;
        if (m < 0) m += nxu;
        int ix = 1 + m;
        double xgu = c.xmin + c.glxu * (double)(ix - 1);
        double x2 = xgu - xi;
        double px0 = (x2 - c.ellx * f_dint(x2 * c.hlxi)) / dx;
        double y2 = yi + px0 * dy;
        int iy = 2 + f_int(c.glyui * (y2 - c.elly * f_dint(y2 * c.hlyi) - c.ymin));
        if (iy >= 2 && iy <= nyu) red_add_s32(&J[(long long)(ix - 1) * nyu + (iy - 1)], jump);
      }
    }
  }
}

__global__ void k_u_lbot(const int *__restrict__ ljx, int *__restrict__ J, int nxu, int nyu) {
  CASL_PDL_ENTRY();
  __shared__ int warp_tot[32];
  __shared__ int carry;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  for (int base = 0; base < nxu; base += blockDim.x) {
    int i = base + threadIdx.x;
    int v = i < nxu ? ljx[i] : 0;
    int x = warp_incl_scan(v);
    if (lane == 31) warp_tot[wid] = x;
    __syncthreads();
    if (wid == 0) {
      int t = lane < nw ? warp_tot[lane] : 0;
      t = warp_incl_scan(t);
      if (lane < nw) warp_tot[lane] = t;
    }
    __syncthreads();
    int incl = x + (wid > 0 ? warp_tot[wid - 1] : 0) + carry;
    if (i < nxu) J[(long long)i * nyu] = incl - v;
    __syncthreads();
    if (threadIdx.x == blockDim.x - 1) carry = incl;
    __syncthreads();
  }
}

// column sweep (congen.f90:419-423) with the column sums for the mean
__global__ void k_u_colscan(int *__restrict__ J, int nxu, int nyu,
                            unsigned long long *__restrict__ total) {
  CASL_PDL_ENTRY();
  int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  int lane = threadIdx.x & 31;
  if (warp >= nxu) return;
  int *col = J + (long long)warp * nyu;
  int carry = 0;
  long long s = 0;
  for (int base = 0; base < nyu; base += 32) {
    int x = warp_incl_scan(col[base + lane]) + carry;
    col[base + lane] = x;
    s += x;
    carry = __shfl_sync(0xffffffffu, x, 31);
  }
  for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  if (lane == 0) atomicAdd(total, (unsigned long long)s);
}

struct LevInfo {
  int levbeg, levend;
  double qjump, qoff, qjumpi;
};

__device__ __forceinline__ double qtmp_of(int lev, const LevInfo &li) {
  return ((double)lev - 0.5) * li.qjump - li.qoff;
}

// Largest level l whose contour value qtmp(l) = (l - 1/2) qjump - qoff is
// <= v.  qtmp is increasing in l (also as rounded), so an edge with end
// values lo < hi crosses exactly the levels c(lo) < l <= c(hi): those where
// the reference's sign(qa - qtmp) differs at the two ends (congen.f90:205-212).
// The index is wanted within 0..65535 (the caller clips it), so the steps stop
// beyond both ends: they end for a qjump of zero or a value that is not finite.
__device__ __forceinline__ int level_steps(int l, double v, const LevInfo &li) {
  l = min(max(l, -1), 65536);
  while (l < 65536 && qtmp_of(l + 1, li) <= v) l++;
  while (l >= 0 && qtmp_of(l, li) > v) l--;
  return l;
}
__device__ __forceinline__ int level_index(double v, const LevInfo &li) {
  return level_steps((int)floor((v + li.qoff) * li.qjumpi + 0.5), v, li);
}

// level_index with the exact checks only near a level boundary: the estimate
// y = (v + qoff)/qjump carries a rounding error of a few units of 1e-16
// relative (it is at most 65536 + nlevm), as do the qtmp values, so where y
// lies farther than 1e-6 from a half-integer the nearest integer is the
// level; anything else (and a non-finite v) takes level_index's steps.  The
// nearest integer is the low word of y + 1.5 * 2^52: the conversions and the
// floor it takes the place of run at a quarter of the FP64 rate.  (An y past
// an int's range would give a wrong code; the levels' range is then refused.)
__device__ __forceinline__ int level_index_fast(double v, const LevInfo &li) {
  const double big = 6755399441055744.0;
  const double y = (v + li.qoff) * li.qjumpi, t = y + big;
  if (fabs(y - (t - big)) < 0.5 - 1.0e-6) return __double2loint(t);
  return level_steps((int)floor(y + 0.5), v, li);
}
__device__ __forceinline__ unsigned int level_code(double v, const LevInfo &li) {
  return (unsigned int)min(max(level_index_fast(v, li), 0), 65535);
}
// (double)i by an integer operation and one subtraction, exact
__device__ __forceinline__ double int_as_double(int i) {
  return __hiloint2double(0x43300000, i ^ (int)0x80000000) - 4503601774854144.0;
}

// One element of the ultra-fine field: (L*qjump - qavg) + bilinear residual,
// or the bilinear residual alone; pxf, pyf is the point's place in its coarse
// cell (cell_part), q00..q11 the cell's corner values.  Per element the
// expression and its order are the reference's (congen.f90:45-61 on
// con2ugrid's field).  The field kernel and the crossing geometry both
// evaluate the field here, so the crossing positions are computed from the
// very values the crossings were found on.
__device__ __forceinline__ double ufield_elem(int lv, double pxf, double pyf, double q00, double q10,
                                              double q01, double q11, double qjump, double qavg,
                                              int have_contours) {
  const double pxc = 1.0 - pxf, pyc = 1.0 - pyf;
  const double w00 = pyc * pxc, w10 = pyf * pxc, w01 = pyc * pxf, w11 = pyf * pxf;
  if (have_contours) {
    double v = int_as_double(lv) * qjump - qavg;
    return v + w00 * q00 + w10 * q10 + w01 * q01 + w11 * q11;
  }
  return w00 * q00 + w10 * q10 + w01 * q01 + w11 * q11;
}
// a point's place in its coarse cell: (place - 1)/16, exact
__device__ __forceinline__ double cell_part(int place) { return (1.0 / 16.0) * (double)(place - 1); }
__device__ __forceinline__ double ufield_qavg(const unsigned long long *lsum, double qjump,
                                              int have_contours, int nxu, int nyu) {
  return have_contours ? qjump * ((double)(long long)(*lsum) / ((double)nxu * (double)nyu)) : 0.0;
}
// the field at the 1-based ultra-fine point (ix, iy)
struct UField {
  const int *L;
  const unsigned long long *lsum;
  const double *qq;
  double qjump;
  int have;
  double bnc;  // beta != 0 without contours: beta*ygu(iy) is added (econgen.f90:94-110)
};
__device__ __forceinline__ double ufield_at(const UField &u, double qavg, int ix, int iy,
                                            const Consts &c) {
  const int n = c.nx;
  const int ixx = (ix - 1) / 16, iyy = (iy - 1) / 16;
  const int ix0 = 1 + ixx, ix1 = 2 + ixx - n * (ix0 / n), ixf = ix - 16 * ixx;
  const int iy0 = 1 + iyy, iy1 = 2 + iyy - n * (iy0 / n), iyf = iy - 16 * iyy;
  const double q00 = u.qq[(long long)(ix0 - 1) * n + iy0 - 1];
  const double q10 = u.qq[(long long)(ix0 - 1) * n + iy1 - 1];
  const double q01 = u.qq[(long long)(ix1 - 1) * n + iy0 - 1];
  const double q11 = u.qq[(long long)(ix1 - 1) * n + iy1 - 1];
  const int lv = u.have ? u.L[(long long)(ix - 1) * c.nyu + iy - 1] : 0;
  const double v = ufield_elem(lv, cell_part(ixf), cell_part(iyf), q00, q10, q01, q11, u.qjump, qavg, u.have);
  return u.bnc != 0.0 ? v + u.bnc * (c.ymin + c.glyu * (double)(iy - 1)) : v;
}

// The ultra-fine field, one thread per run of 16 rows of a column: the run
// lies in one coarse cell in y, so the four coarse values are gathered once;
// the levels come in as 16-byte vectors.  Out go the field itself (qa, when
// asked for) and/or its level code lc = level_index(v) clipped to
// [0, 65535], with the field's extremes.  qtmp depends only on qjump and
// nlevm, so the code is known before the level range is.
__global__ void __launch_bounds__(256, 4) k_u_field(const int *__restrict__ L, const unsigned long long *__restrict__ lsum,
                          const double *__restrict__ qq, double qjump, int have_contours,
                          LevInfo lq, double *__restrict__ qa, unsigned short *__restrict__ lc,
                          unsigned long long *__restrict__ ext, Consts c, double bnc) {
  CASL_PDL_ENTRY();
  const int nxu = c.nxu, nyu = c.nyu, n = c.nx;
  const long long nruns = (long long)nxu * (nyu / 16);
  const double qavg = ufield_qavg(lsum, qjump, have_contours, nxu, nyu);
  double mx = -1.0e308, mn = 1.0e308, l1 = 0.0;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < nruns;
       t += (long long)gridDim.x * blockDim.x) {
    const int iyy = (int)(t % (nyu / 16)), ix = (int)(t / (nyu / 16)) + 1;
    const int ixx = (ix - 1) / 16;
    const int ix0 = 1 + ixx, ix1 = 2 + ixx - n * (ix0 / n), ixf = ix - 16 * ixx;
    const int iy0 = 1 + iyy, iy1 = 2 + iyy - n * (iy0 / n);
    const double q00 = qq[(long long)(ix0 - 1) * n + iy0 - 1], q10 = qq[(long long)(ix0 - 1) * n + iy1 - 1];
    const double q01 = qq[(long long)(ix1 - 1) * n + iy0 - 1], q11 = qq[(long long)(ix1 - 1) * n + iy1 - 1];
    if (ixf == 1) l1 += fabs(q00);  // every residual point once
    const long long base = (long long)(ix - 1) * nyu + 16LL * iyy;
    const double pxf = cell_part(ixf);
    // the run in two halves of 8 points (fewer live registers)
#pragma unroll 1
    for (int hf = 0; hf < 2; hf++) {
      int lv[8];
      if (have_contours) {
        const int4 *l4 = reinterpret_cast<const int4 *>(L + base) + 2 * hf;
        const int4 q0 = l4[0], q1 = l4[1];
        lv[0] = q0.x; lv[1] = q0.y; lv[2] = q0.z; lv[3] = q0.w;
        lv[4] = q1.x; lv[5] = q1.y; lv[6] = q1.z; lv[7] = q1.w;
      } else {
#pragma unroll
        for (int k = 0; k < 8; k++) lv[k] = 0;
      }
      const double pyh = 0.5 * hf;  // the half's first point
      unsigned int code[4];
#pragma unroll
      for (int k = 0; k < 4; k++) {
        double out[2];
#pragma unroll
        for (int h = 0; h < 2; h++) {
          const int iyf = 8 * hf + 2 * k + h;  // 0-based place in the run
          double v = ufield_elem(lv[2 * k + h], pxf, pyh + (2 * k + h) * (1.0 / 16.0), q00, q10, q01, q11,
                                 qjump, qavg, have_contours);
          if (bnc != 0.0) v = v + bnc * (c.ymin + c.glyu * (double)(16 * iyy + iyf));
          out[h] = v;
          mx = v > mx ? v : mx;  // (fmax and fmin take twice the instructions)
          mn = v < mn ? v : mn;
        }
        if (qa) reinterpret_cast<double2 *>(qa + base)[4 * hf + k] = make_double2(out[0], out[1]);
        if (lc) {
          code[k] = level_code(out[0], lq) | level_code(out[1], lq) << 16;
        }
      }
      if (lc)
        reinterpret_cast<uint4 *>(lc + base)[hf] = make_uint4(code[0], code[1], code[2], code[3]);
    }
  }
  // extremes and sum of |residual|: ext[0] the largest value's ordered word,
  // ext[1] the complement of the smallest's, ext[2] the sum (a double), all 0
  // on entry
  __shared__ double a[8], b[8], w[8];
  for (int o = 16; o > 0; o >>= 1) {
    mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    mn = fmin(mn, __shfl_xor_sync(0xffffffffu, mn, o));
    l1 += __shfl_xor_sync(0xffffffffu, l1, o);
  }
  if ((threadIdx.x & 31) == 0) {
    a[threadIdx.x >> 5] = mx;
    b[threadIdx.x >> 5] = mn;
    w[threadIdx.x >> 5] = l1;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int k = 1; k < 8; k++) {
      mx = fmax(mx, a[k]);
      mn = fmin(mn, b[k]);
      l1 += w[k];
    }
    atomicMax(&ext[0], ordered_word(mx));
    atomicMax(&ext[1], ~ordered_word(mn));
    if (!have_contours) atomicAdd(reinterpret_cast<double *>(ext + 2), l1);
  }
}

// ---------------------------------------------------------------------------
// beta != 0 (econgen.f90:27-488): the grid extended in y
// ---------------------------------------------------------------------------
// PV on a beta-plane is not periodic in y: the periodic image of row iy0 one
// box up carries an extra beta*Ly.  The field is extended over rows
// iymin..iymax, row iy taking the values of basic row iy0 = 1 + mod(iy-1,
// nyu) plus bfac*(iy - iy0), bfac = beta*glyu; contours are traced on the
// extended grid and only one periodic image of each is kept.
struct ExtGrid {
  int iymin, iymax, nby;       // nby: boxes below the basic one (econgen.f90:217)
  double bfac;
};
__device__ __forceinline__ int ext_row0(const ExtGrid &g, int iy, int nyu) {
  return iy < 1 ? 1 + (g.nby * nyu + iy - 1) % nyu : (iy > nyu ? 1 + (iy - 1) % nyu : iy);
}
// Minimum and maximum of the field along every basic row (econgen.f90:
// 114-129) as ordered words, the minimum's complemented, both 0 on entry: a
// block takes 16 rows (one coarse cell) of 512 columns, a thread two columns'
// runs of them.  (One block per 16 rows, all columns: 256 blocks at 256^2 and
// the corner values read at every point, 74 us; so 48.)
__global__ void __launch_bounds__(256) k_u_rowmm(UField uf, Consts c,
                                                 unsigned long long *__restrict__ rmin,
                                                 unsigned long long *__restrict__ rmax) {
  CASL_PDL_ENTRY();
  const int nxu = c.nxu, nyu = c.nyu, n = c.nx;
  const double qavg = ufield_qavg(uf.lsum, uf.qjump, uf.have, nxu, nyu);
  const int iyy = blockIdx.x, iy0 = 1 + iyy, iy1 = 2 + iyy - n * (iy0 / n);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  double mn[16], mx[16];
#pragma unroll
  for (int k = 0; k < 16; k++) {
    mn[k] = 1.0e308;
    mx[k] = -1.0e308;
  }
#pragma unroll 1
  for (int h = 0; h < 2; h++) {
    const int ix = (2 * blockIdx.y + h) * 256 + threadIdx.x + 1, ixx = (ix - 1) / 16;
    const int ix0 = 1 + ixx, ix1 = 2 + ixx - n * (ix0 / n);
    const double *q0 = uf.qq + (long long)(ix0 - 1) * n, *q1 = uf.qq + (long long)(ix1 - 1) * n;
    const double q00 = q0[iy0 - 1], q10 = q0[iy1 - 1], q01 = q1[iy0 - 1], q11 = q1[iy1 - 1];
    const double pxf = cell_part(ix - 16 * ixx);
    const int4 *l4 = reinterpret_cast<const int4 *>(uf.L + (long long)(ix - 1) * nyu + 16LL * iyy);
#pragma unroll
    for (int k = 0; k < 16; k++) {
      int4 l = make_int4(0, 0, 0, 0);
      if (uf.have) l = l4[k / 4];
      const int lv = k % 4 == 0 ? l.x : (k % 4 == 1 ? l.y : (k % 4 == 2 ? l.z : l.w));
      double v = ufield_elem(lv, pxf, k * (1.0 / 16.0), q00, q10, q01, q11, uf.qjump, qavg, uf.have);
      if (uf.bnc != 0.0) v = v + uf.bnc * (c.ymin + c.glyu * (double)(16 * iyy + k));
      mn[k] = v < mn[k] ? v : mn[k];
      mx[k] = v > mx[k] ? v : mx[k];
    }
  }
  // across the warp, each step with half the rows: lanes 2k and 2k+1 end with
  // row k
#pragma unroll
  for (int o = 16, m = 8; m >= 1; o >>= 1, m >>= 1) {
    const bool hi = lane & o;
#pragma unroll
    for (int k = 0; k < m; k++) {
      const double a = __shfl_xor_sync(0xffffffffu, hi ? mn[k] : mn[k + m], o);
      const double b = __shfl_xor_sync(0xffffffffu, hi ? mx[k] : mx[k + m], o);
      const double ka = hi ? mn[k + m] : mn[k], kb = hi ? mx[k + m] : mx[k];
      mn[k] = a < ka ? a : ka;
      mx[k] = b > kb ? b : kb;
    }
  }
  __shared__ double smn[8][16], smx[8][16];
  {
    const double a = __shfl_xor_sync(0xffffffffu, mn[0], 1), b = __shfl_xor_sync(0xffffffffu, mx[0], 1);
    if (!(lane & 1)) {
      smn[w][lane >> 1] = a < mn[0] ? a : mn[0];
      smx[w][lane >> 1] = b > mx[0] ? b : mx[0];
    }
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    const int k = threadIdx.x & 15;
    const bool up = threadIdx.x >= 16;
    double a = up ? smx[0][k] : smn[0][k];
    for (int q = 1; q < 8; q++) {
      const double x = up ? smx[q][k] : smn[q][k];
      a = up == (x > a) ? x : a;
    }
    if (up)
      atomicMax(&rmax[16 * iyy + k], ordered_word(a));
    else
      atomicMax(&rmin[16 * iyy + k], ~ordered_word(a));
  }
}

// Level codes of the extended grid, column by column (ld codes each), rows
// iymin..iymax: the basic rows' codes, and in the extension the level index
// of qa(iy0) + bfac*(iy - iy0), the value rounded once as the reference's
// x-line scan forms it (econgen.f90:247-258).  A block takes 256 rows of the
// 16 columns of one coarse cell, a thread one row: its corner values and
// offset are formed once.  (A thread a point, with a 64-bit division, four
// gathers and the full level search at each: 185 us at 256^2; so 50.)
__global__ void __launch_bounds__(256) k_u_ext(UField uf, ExtGrid g, LevInfo li, Consts c,
                                               const unsigned short *__restrict__ lc, long long ld,
                                               unsigned short *__restrict__ le) {
  CASL_PDL_ENTRY();
  const int nxu = c.nxu, nyu = c.nyu, n = c.nx, nr = g.iymax - g.iymin + 1;
  const int r = blockIdx.x * 256 + threadIdx.x, ixx = blockIdx.y;
  if (r >= nr) return;
  const int iy = g.iymin + r;
  unsigned short *o = le + 16LL * ixx * ld + r;
  if (iy >= 1 && iy <= nyu) {
    const unsigned short *s = lc + 16LL * ixx * nyu + iy - 1;
#pragma unroll
    for (int k = 0; k < 16; k++) o[k * ld] = s[(long long)k * nyu];
    return;
  }
  const double qavg = ufield_qavg(uf.lsum, uf.qjump, uf.have, nxu, nyu);
  const int yb = ext_row0(g, iy, nyu), iyy = (yb - 1) / 16;
  const double add = g.bfac * (double)(iy - yb), pyf = cell_part(yb - 16 * iyy);
  const double yn = uf.bnc != 0.0 ? uf.bnc * (c.ymin + c.glyu * (double)(yb - 1)) : 0.0;
  const int ix0 = 1 + ixx, ix1 = 2 + ixx - n * (ix0 / n);
  const int iy0 = 1 + iyy, iy1 = 2 + iyy - n * (iy0 / n);
  const double *q0 = uf.qq + (long long)(ix0 - 1) * n, *q1 = uf.qq + (long long)(ix1 - 1) * n;
  const double q00 = q0[iy0 - 1], q10 = q0[iy1 - 1], q01 = q1[iy0 - 1], q11 = q1[iy1 - 1];
  const int *L = uf.L + 16LL * ixx * nyu + yb - 1;
#pragma unroll 4
  for (int k = 0; k < 16; k++) {
    const int lv = uf.have ? L[(long long)k * nyu] : 0;
    double v = ufield_elem(lv, cell_part(k + 1), pyf, q00, q10, q01, q11, uf.qjump, qavg, uf.have);
    if (uf.bnc != 0.0) v = v + yn;
    o[k * ld] = (unsigned short)level_code(v + add, li);
  }
}

// One periodic image per contour (econgen.f90:238-246): bit 0 of flags[k]
// is set when a crossing of contour k lies below ymin, bit 1 when one lies
// below ymax; k is kept when bit 0 is clear and bit 1 set.
// (A contour's crossings are consecutive: a warp that lies in one contour
// combines its bits, and bits already there are not set again; an atomic per
// crossing took 435 us at 256^2, this 40.)
__global__ void k_ec_flags(const double *__restrict__ yw, const int *__restrict__ cidw, long long N,
                           Consts c, int *__restrict__ flags) {
  CASL_PDL_ENTRY();
  for (long long b = blockIdx.x * (long long)blockDim.x; b < N; b += (long long)gridDim.x * blockDim.x) {
    const long long w = b + threadIdx.x;
    const bool in = w < N;
    const double y = in ? yw[w] : 0.0;
    const int k = in ? cidw[w] : -1;
    int f = in ? (y < c.ymin ? 1 : 0) | (y < c.ymax ? 2 : 0) : 0;
    const int k0 = __shfl_sync(0xffffffffu, k, 0);
    if (__all_sync(0xffffffffu, k == k0)) {
      f = __reduce_or_sync(0xffffffffu, f);
      if (threadIdx.x & 31) f = 0;
    }
    if (f && (__ldcg(&flags[k]) & f) != f) atomicOr(&flags[k], f);
  }
}
__global__ void k_ec_keep(const int *__restrict__ flags, const int *__restrict__ clen, int C,
                          int *__restrict__ klen, int *__restrict__ kone) {
  CASL_PDL_ENTRY();
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < C; k += gridDim.x * blockDim.x) {
    const bool keep = !(flags[k] & 1) && (flags[k] & 2);
    klen[k] = keep ? clen[k] : 0;
    kone[k] = keep ? 1 : 0;
  }
}
// The kept contours' crossings, y folded into [ymin, ymax) by
// mod(y + yoff, elly) + ymin (econgen.f90:249-252), and their contour list.
__global__ void k_ec_compact(const double *__restrict__ xw, const double *__restrict__ yw,
                             const int *__restrict__ cidw, long long N, const int *__restrict__ coff,
                             const int *__restrict__ klen, const int *__restrict__ koff,
                             const int *__restrict__ kidx, Consts c, double yoff,
                             double *__restrict__ xw2, double *__restrict__ yw2,
                             int *__restrict__ cidw2) {
  CASL_PDL_ENTRY();
  for (long long w = blockIdx.x * (long long)blockDim.x + threadIdx.x; w < N;
       w += (long long)gridDim.x * blockDim.x) {
    const int k = cidw[w];
    if (!klen[k]) continue;
    const long long d = koff[k] + (w - coff[k]);
    xw2[d] = xw[w];
    yw2[d] = fmod(yw[w] + yoff, c.elly) + c.ymin;
    cidw2[d] = kidx[k];
  }
}
__global__ void k_ec_contours(const int *__restrict__ clen, const int *__restrict__ clevt, int C,
                              const int *__restrict__ klen, const int *__restrict__ koff,
                              const int *__restrict__ kidx, int *__restrict__ cs2,
                              int *__restrict__ len2, int *__restrict__ lev2) {
  CASL_PDL_ENTRY();
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < C; k += gridDim.x * blockDim.x) {
    if (!klen[k]) continue;
    const int j = kidx[k];
    cs2[j] = koff[k];
    len2[j] = clen[k];
    lev2[j] = clevt[k];
  }
}

__global__ void k_set_counts2(Scalars *s, const int *cnt) {
  CASL_PDL_ENTRY();
  s->nq = cnt[0];
  s->nptq = cnt[1];
}
__global__ void k_out_contours(const int *__restrict__ ocs, const int *__restrict__ olen,
                               const int *__restrict__ olev, int nq, int *__restrict__ i1q,
                               int *__restrict__ i2q, int *__restrict__ npq,
                               int *__restrict__ indq) {
  CASL_PDL_ENTRY();
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < nq; j += gridDim.x * blockDim.x) {
    i1q[j] = ocs[j];
    i2q[j] = ocs[j] + olen[j] - 1;
    npq[j] = olen[j];
    indq[j] = olev[j];
  }
}
__global__ void k_out_links(const int *__restrict__ ocs, const int *__restrict__ olen, int nq,
                            int npt, int *__restrict__ nextq) {
  CASL_PDL_ENTRY();
  for (long long b = blockIdx.x * (long long)CC_CHUNK; b < npt; b += (long long)gridDim.x * CC_CHUNK) {
    chunk_contours(ocs, nq, b);
    for (int i = (int)b + threadIdx.x; i < min((long long)npt, b + CC_CHUNK); i += blockDim.x) {
      const int j = chunk_contour_of(ocs, nq, i);
      nextq[i] = i + 1 < ocs[j] + olen[j] ? i + 1 : ocs[j];
    }
  }
}


}  // namespace casl

#include "trace.cuh"

namespace casl {

static inline int gsz(long long work) {
  long long g = (work + 255) / 256;
  if (g < 1) g = 1;
  if (g > 148 * 32) g = 148 * 32;
  return (int)g;
}

#define RC_TRY(x)        \
  do {                   \
    int _r = (x);        \
    if (_r) return _r;   \
  } while (0)

// Small device results for the host: all of them, and the error word, land in
// pinned memory behind one wait.  Copies to the caller's own variables are
// staged by the driver one after the other, 20 us each.  What does not fit
// goes to its destination directly.  Returns the error word.
struct ReadItem {
  void *dst;
  const void *src;
  size_t bytes;
};
static int read_back(casl_handle *h, std::initializer_list<ReadItem> items) {
  constexpr size_t cap = 256 << 10;
  cudaStream_t st = h->stream;
  if (!h->hpin && cudaMallocHost(&h->hpin, cap) != cudaSuccess) {
    cudaGetLastError();
    h->hpin = nullptr;
  }
  int err = 0;
  size_t off = 16;  // the error word lies first
  std::vector<size_t> at;
  for (const ReadItem &r : items) {
    const bool fits = h->hpin && off + r.bytes <= cap;
    at.push_back(fits && r.bytes ? off : 0);
    if (!r.bytes) continue;
    CASL_CUDA_TRY(cudaMemcpyAsync(fits ? h->hpin + off : r.dst, r.src, r.bytes,
                                  cudaMemcpyDeviceToHost, st));
    if (fits) off += (r.bytes + 15) / 16 * 16;
  }
  CASL_CUDA_TRY(cudaMemcpyAsync(h->hpin ? (void *)h->hpin : &err, &h->scal->error, sizeof(int),
                                cudaMemcpyDeviceToHost, st));
  CASL_CUDA_TRY(cudaStreamSynchronize(st));
  if (h->hpin) memcpy(&err, h->hpin, sizeof(int));
  size_t k = 0;
  for (const ReadItem &r : items) {
    if (at[k]) memcpy(r.dst, h->hpin + at[k], r.bytes);
    k++;
  }
  return err;
}

// l1norm (generic.f90:180-194) of the residual, summed as the reference does
static int l1_host(casl_handle *h, const double *qq, double *l1) {
  std::vector<double> hq((size_t)h->c.nx * h->c.ny);
  CASL_CUDA_TRY(cudaMemcpyAsync(hq.data(), qq, hq.size() * sizeof(double), cudaMemcpyDeviceToHost, h->stream));
  CASL_CUDA_TRY(cudaStreamSynchronize(h->stream));
  *l1 = 0.0;
  for (double v : hq) *l1 += fabs(v);
  return CASL_OK;
}

template <class Rel>
static int launch_walk(casl_handle *h, const TrArgs &ta, int ntile, int nslice) {
  static std::atomic<unsigned long long> configured{0};  // a bit per device
  const unsigned long long bit = 1ULL << (h->device & 63);
  if (!(configured.load() & bit)) {
    CASL_CUDA_TRY(cudaFuncSetAttribute(k_tr_walk<Rel>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)sizeof(TrSmem<Rel>)));
    configured.fetch_or(bit);
  }
  CASL_K(k_tr_walk<Rel>, dim3(ntile, nslice), TR_NT, sizeof(TrSmem<Rel>), h->stream)(ta);
  return CASL_OK;
}

int recontour_dev(casl_handle *h, const double *qq) {
  cudaStream_t st = h->stream;
  const Consts &c = h->c;
  const int nxu = c.nxu, nyu = c.nyu;
  const long long NU = (long long)nxu * nyu;
  const double qjump = h->qjump;
  const int have = h->nptq > 0 && h->nq > 0;
  // beta != 0 recontours as econgen.f90 does (the reference's ecaps build):
  // beta*Ly must be a whole number of contour intervals (econgen.f90:52-60,
  // where the reference stops)
  const bool econ = c.beffect != 0;
  const double bfac = c.beta * c.glyu, ppvdif = c.beta * c.elly;
  if (econ) {
    const double brat = ppvdif * (1.0 / qjump);
    if (!(fabs(brat - (double)llround(brat)) <= 1.0e-7)) return CASL_EINVAL;
  }
  const double bnc = econ && !have ? c.beta : 0.0;
  cudaMemsetAsync(&h->scal->error, 0, sizeof(int), st);
  Trace tr;
  tr.begin(st, "start");
  struct Flush {
    Trace &t;
    ~Flush() { t.flush("recontour"); }
  } flush_at_exit{tr};

  // --- 1. ultra-fine field ---------------------------------------------------
  auto set_empty = [&]() -> int {
    h->nq = h->nptq = 0;
    h->hscal->nq = h->hscal->nptq = 0;
    int z[2] = {0, 0};
    CASL_CUDA_TRY(cudaMemcpyAsync(&h->scal->nq, z, 2 * sizeof(int), cudaMemcpyHostToDevice, st));
    CASL_CUDA_TRY(cudaStreamSynchronize(st));
    return CASL_OK;
  };
  // nothing to contour if l1norm (generic.f90:180-194) of the full field is
  // ~0.  k_u_field sums it beside the level codes; with no interval to speak
  // of (a field of zeros has none) the codes mean nothing and the host sums.
  if (!have && !econ && !(qjump > 1.0e-200)) {
    double l1 = 0.0;
    RC_TRY(l1_host(h, qq, &l1));
    if (c.garea * l1 < c.small) return set_empty();
  }
  // Field memory: level codes + integer levels + per-chunk crossing counts;
  // kept for the whole call.
  const long long nchunks_f = 2 * NU / 16;
  size_t need_field = (size_t)NU * 6 + (size_t)nchunks_f * 8 + (size_t)nxu * 4 +
                      (size_t)nyu * 16 + ((size_t)64 << 20);
  if (int rc = ensure_scratch(h, need_field)) {
    // a field of zeros needs no memory
    double l1 = 1.0;
    if (!have && !econ) RC_TRY(l1_host(h, qq, &l1));
    if (c.garea * l1 < c.small) return set_empty();
    return rc;
  }
  Arena ar{(char *)h->sx, h->sx_bytes, 0};
  unsigned short *lc = ar.get<unsigned short>(NU);
  int *Lu = ar.get<int>(NU);
  int *ljx = ar.get<int>(nxu);
  // level sum; k_u_field's results; k_cr_count's word
  unsigned long long *lsum = ar.get<unsigned long long>(5);
  unsigned long long *rmn = ar.get<unsigned long long>(2 * nyu), *rmx = rmn + nyu;
  int *dtot = ar.get<int>(16);
  if (ar.failed) return CASL_ENOMEM;
  CASL_CUDA_TRY(cudaMemsetAsync(lsum, 0, 5 * sizeof(unsigned long long), st));
  if (have) {
    CASL_CUDA_TRY(cudaMemsetAsync(Lu, 0, (size_t)NU * sizeof(int), st));
    CASL_CUDA_TRY(cudaMemsetAsync(ljx, 0, (size_t)nxu * sizeof(int), st));
    tr.point("u_memset");
    CASL_K(k_u_scatter, gsz(h->nptq), 256, 0, st)(h->xq, h->yq, h->nextq, h->nptq, qjump, Lu, ljx, c,
                                              &h->scal->error);
    tr.point("u_scatter");
    CASL_K(k_u_lbot, 1, 1024, 0, st)(ljx, Lu, nxu, nyu);
    CASL_K(k_u_colscan, (nxu * 32 + 255) / 256, 256, 0, st)(Lu, nxu, nyu, lsum);
    tr.point("u_colscan");
  }
  // qtmp(l) = (l - 1/2) qjump - qoff with qoff = qjump*nlevm (congen.f90:156-173)
  LevInfo li;
  li.qjump = qjump;
  li.qjumpi = 1.0 / qjump;
  li.qoff = qjump * (double)h->p.nlevm;
  li.levbeg = li.levend = 0;
  CASL_K(k_u_field, 4096, 256, 0, st)(Lu, lsum, qq, qjump, have, li, nullptr, lc, lsum + 1, c, bnc);
  RC_TRY(check_launch(h));
  double qamax = 0.0, qamin = 0.0;
  if (!econ) {
    unsigned long long ext[3];
    RC_TRY(read_back(h, {{ext, lsum + 1, sizeof(ext)}}));
    qamax = from_ordered(ext[0]);
    qamin = from_ordered(~ext[1]);
    if (!have) {
      // the device sums in another order: close to the line the host decides
      double l1;
      memcpy(&l1, &ext[2], 8);
      if (fabs(c.garea * l1 - c.small) <= 1.0e-9 * c.small) RC_TRY(l1_host(h, qq, &l1));
      if (c.garea * l1 < c.small) return set_empty();
    }
  }
  tr.point("field");
  const UField uf{have ? Lu : nullptr, lsum, qq, qjump, have, bnc};
  // beta != 0: the extent of the y-extended grid (econgen.f90:112-171), on
  // the host from the rows' minima and maxima
  ExtGrid eg{};
  if (econ) {
    const FillJob z[1] = {{rmn, 4LL * nyu, 0u}};
    RC_TRY(fill_words(st, z, 1));
    CASL_K(k_u_rowmm, dim3(nyu / 16, nxu / 512), 256, 0, st)(uf, c, rmn, rmx);
    std::vector<double> qqmin(nyu + 2), qqmax(nyu + 2);
    std::vector<unsigned long long> mm(2 * nyu);
    RC_TRY(read_back(h, {{mm.data(), rmn, mm.size() * 8}}));
    for (int iy = 0; iy < nyu; iy++) {
      qqmin[iy + 1] = from_ordered(~mm[iy]);
      qqmax[iy + 1] = from_ordered(mm[nyu + iy]);
    }
    qqmin[nyu + 1] = qqmin[1] + ppvdif;
    qqmax[nyu + 1] = qqmax[1] + ppvdif;
    qamin = qqmin[1];
    qamax = qqmax[1];
    for (int iy = 2; iy <= nyu + 1; iy++) {
      qamin = std::min(qamin, qqmin[iy]);
      qamax = std::max(qamax, qqmax[iy]);
    }
    // the lowest and highest rows that meet a level of the basic box; the
    // reference assumes fewer than 100 periodic boxes
    const int levmin = (int)(qamin * li.qjumpi - 0.5);
    double qlev = ((double)levmin + 0.5) * qjump;
    int iy = 1;
    for (;;) {
      iy = iy - 1;
      if (iy < -100 * nyu) return CASL_ECAPACITY;
      const int iy0 = 1 + (100 * nyu + iy - 1) % nyu;
      if (bfac * (double)(iy - iy0) + qqmax[iy0] <= qlev) break;
    }
    eg.iymin = iy;
    const int levmax = (int)(qamax * li.qjumpi + 0.5);
    qlev = ((double)levmax - 0.5) * qjump;
    iy = nyu + 1;
    for (;;) {
      iy = iy + 1;
      if (iy > 101 * nyu) return CASL_ECAPACITY;
      const int iy0 = 1 + (iy - 1) % nyu;
      if (bfac * (double)(iy - iy0) + qqmin[iy0] >= qlev) break;
    }
    eg.iymax = iy;
    eg.nby = 1 - eg.iymin / nyu;
    eg.bfac = bfac;
    // extended grids of 2^32 points and more are refused, as they were when
    // boxes had 32-bit numbers (10 GB of codes and counts; crossings are
    // counted in an int)
    if ((long long)nxu * (eg.iymax - eg.iymin + 2) >= (1LL << 32)) return CASL_ECAPACITY;
  }
  // --- 2. levels (congen.f90:156-173; econgen.f90:131-134) -------------------
  li.levbeg = (int)((li.qoff + qamin) * li.qjumpi + 0.5) + 1;
  li.levend = (int)((li.qoff + qamax) * li.qjumpi + 0.5);
  // the level codes hold 0..65535: levels must lie inside
  if (li.levbeg <= li.levend && (li.levbeg < 1 || li.levend > 65534)) return CASL_ECAPACITY;
  if (li.levbeg > li.levend) return set_empty();
  const int nlev = li.levend - li.levbeg + 1;

  tr.point("levels");
  // --- 3. crossings in reference order ----------------------------------------
  // beta != 0: the extended grid's codes and edges
  const int nye = econ ? eg.iymax - eg.iymin + 1 : 0;
  CrGrid cg{};
  cg.nxu = nxu;
  cg.periodic = !econ;
  cg.nrow = econ ? nye : nyu;
  cg.ner = cg.nbr = econ ? nye - 1 : nyu;
  cg.nseg = (cg.ner + 15) / 16;
  cg.ylo = econ ? 1 : 0;
  cg.nyl = econ ? nye - 2 : nyu;
  cg.ld = econ ? ((long long)nye + 255) / 256 * 256 : nyu;
  cg.ncx = (long long)nxu * cg.nseg;
  cg.cmin = li.levbeg - 1;
  cg.cmax = li.levend;
  cg.lc = lc;
  const long long nchunks = cr_chunks(cg);
  int *ccnt, *coffs, *tmpi;
  if (econ) {
    // codes and chunk counts in a buffer of their own (the field arena is
    // sized before the extension is known)
    const size_t bcodes = ((size_t)nxu * cg.ld * 2 + 255) / 256 * 256;
    const size_t need = bcodes + (size_t)nchunks * 8 + (size_t)(scan_tmp_elems(nchunks) + 4) * 4 +
                        ((size_t)1 << 20);
    if (h->sxe_bytes < need) {
      if (h->sxe) cudaFree(h->sxe);
      h->sxe = nullptr;
      h->sxe_bytes = 0;
      CASL_CUDA_TRY(cudaMalloc(&h->sxe, need + need / 2));
      h->sxe_bytes = need + need / 2;
    }
    Arena are{(char *)h->sxe, h->sxe_bytes, 0};
    unsigned short *le = are.get<unsigned short>((size_t)nxu * cg.ld);
    ccnt = are.get<int>(nchunks);
    coffs = are.get<int>(nchunks + 1);
    tmpi = are.get<int>(scan_tmp_elems(nchunks) + 4);
    if (are.failed) return CASL_ENOMEM;
    cg.lc = le;
    CASL_K(k_u_ext, dim3((nye + 255) / 256, c.nx), 256, 0, st)(uf, eg, li, c, lc, cg.ld, le);
  } else {
    ccnt = ar.get<int>(nchunks);
    coffs = ar.get<int>(nchunks + 1);
    tmpi = ar.get<int>(scan_tmp_elems(nchunks) + 4);
    if (ar.failed) return CASL_ENOMEM;
  }
  CASL_K(k_cr_count, (int)((nxu / 128) * (cg.ld / 256)), 256, 0, st)(
      cg, ccnt, reinterpret_cast<int *>(lsum + 4));
  tr.point("cr_count");
  exclusive_scan<int>(st, ccnt, coffs, nchunks, tmpi, dtot);
  // the offset after the last chunk
  CASL_CUDA_TRY(cudaMemcpyAsync(coffs + nchunks, dtot, sizeof(int), cudaMemcpyDeviceToDevice, st));
  int ncr_i = 0, wide = 0;
  RC_TRY(read_back(h, {{&ncr_i, dtot, sizeof(int)}, {&wide, lsum + 4, sizeof(int)}}));
  const long long ncr = ncr_i;
  if (tr.on) fprintf(stderr, "[casl trace] recontour: %lld crossings on %d levels\n", ncr, nlev);
  if (ncr == 0) return set_empty();
  // Per-crossing storage lives in a second arena sized from the count, so
  // that the ultra-fine field in the first one is kept.
  {
    const long long capn = std::max<long long>(ncr * 2, h->npm);
    RC_TRY(ensure_scratch2(h, (size_t)ncr * 448 + (size_t)capn * 32 + ((size_t)64 << 20)));
  }
  Arena ar2{(char *)h->sx2, h->sx2_bytes, 0};
  TrArgs ta{};
  ta.g = cg;
  ta.off = coffs;
  ta.own = ar2.get<int2>(ncr);
  ta.chain = ar2.get<int4>(ncr);
  ta.clev = ar2.get<int>(ncr);
  ta.eidx = ar2.get<int>(ncr);
  ta.eslot = ar2.get<long long>(ncr);
  ta.nchain = dtot + 2;
  ta.nend = dtot + 3;
  ta.cap = (int)ncr;
  ta.err = &h->scal->error;
  if (ar2.failed) return CASL_ENOMEM;
  tr.point("cr_alloc");
  // --- 4. contours followed inside tiles ----------------------------------------
  {
    const FillJob z[1] = {{ta.nchain, 2, 0u}};
    RC_TRY(fill_words(st, z, 1));
  }
  const int ntile = (nxu / TX) * ((cg.nbr + TY - 1) / TY), nslice = tr_slices(ntile, ncr);
  RC_TRY(wide ? launch_walk<unsigned int>(h, ta, ntile, nslice)
              : launch_walk<unsigned short>(h, ta, ntile, nslice));
  RC_TRY(check_launch(h));
  int cnts[2] = {0, 0};
  RC_TRY(read_back(h, {{cnts, ta.nchain, 2 * sizeof(int)}}));
  const int S = cnts[0], nends = cnts[1];
  if (S <= 0) return CASL_EINVAL;
  if (tr.on)
    fprintf(stderr, "[casl trace] tracing: %d chains, %.1f crossings each, %d saddle entries\n", S,
            (double)ncr / S, nends);
  tr.point("trace");
  // --- 5. ranking over the chains -------------------------------------------------
  int *nexts = ar2.get<int>(S), *head = ar2.get<int>(S), *cslot = ar2.get<int>(S);
  int4 *jA = ar2.get<int4>(S), *jB = ar2.get<int4>(S);
  SlSuf *lA = ar2.get<SlSuf>(S), *lB = ar2.get<SlSuf>(S);
  const long long ccap = (long long)S + 2LL * nends;  // contours: cycles and those through saddles
  unsigned long long *key = ar2.get<unsigned long long>(ccap), *key2 = ar2.get<unsigned long long>(ccap);
  int *slot = ar2.get<int>(ccap), *slot2 = ar2.get<int>(ccap), *slen = ar2.get<int>(ccap);
  if (ar2.failed) return CASL_ENOMEM;
  constexpr int MAXR = 18;  // 4^17 windows cover any int count of chains, and one launch to see it
  int *flag = ar2.get<int>(2 * MAXR);
  if (ar2.failed) return CASL_ENOMEM;
  const int gsS = gsz(S);
  int rounds = 1;
  while (rounds < MAXR - 1 && (1LL << (2 * rounds)) < S) rounds++;
  rounds++;
  {
    const FillJob z[2] = {{flag, 2 * MAXR, 0u}, {dtot + 4, 1, 0u}};
    RC_TRY(fill_words(st, z, 2));
  }
  CASL_K(k_ch_init, gsS, 256, 0, st)(ta.chain, ta.own, S, nexts, jA, ta.err);
  for (int it = 0; it < rounds; it++) {
    CASL_K(k_ch_jump1, gsS, 256, 0, st)(jA, S, jB, it, flag);
    std::swap(jA, jB);
  }
  CASL_K(k_ch_list, gsS, 256, 0, st)(nexts, jA, ta.own, ta.chain, S, lA, head);
  for (int it = 0; it < rounds; it++) {
    CASL_K(k_ch_jump2, gsS, 256, 0, st)(lA, S, lB, it, flag + MAXR);
    std::swap(lA, lB);
  }
  if (tr.on) {
    int f[2 * MAXR], ran[2] = {1, 1};
    RC_TRY(read_back(h, {{f, flag, sizeof(f)}}));
    for (int q = 0; q < 2; q++)
      while (ran[q] < rounds && f[q * MAXR + ran[q] - 1]) ran[q]++;
    fprintf(stderr, "[casl trace] ranking: %d and %d of %d launches\n", ran[0], ran[1], rounds);
  }
  CASL_K(k_ch_heads, gsS, 256, 0, st)(head, jA, lA, ta.clev, S, key, slot, slen, cslot, dtot + 4);
  RC_TRY(check_launch(h));
  int C0 = 0;
  std::vector<int> eidx(nends);
  std::vector<long long> eslot(nends);
  RC_TRY(read_back(h, {{&C0, dtot + 4, sizeof(int)},
                       {eidx.data(), ta.eidx, nends * sizeof(int)},
                       {eslot.data(), ta.eslot, nends * sizeof(long long)}}));
  tr.point("ranking");
  // --- 6. lists between saddles: exact simulation of the reference traversal -------
  // Only the crossings entering saddle boxes and the list starts come to the
  // host; everything of size ncr stays on the device.
  int nsad_contours = 0;
  int *listof = nullptr, *d_ladd = nullptr, *d_lslot = nullptr;
  if (nends > 0) {
    std::vector<long long> sad_p(eslot);
    std::sort(sad_p.begin(), sad_p.end());
    sad_p.erase(std::unique(sad_p.begin(), sad_p.end()), sad_p.end());
    const int nsb = (int)sad_p.size();
    // each saddle box is named by its two out-crossings, lower index first
    std::vector<int> slot2h(2 * nsb);
    for (int b = 0; b < nsb; b++) {
      slot2h[2 * b] = (int)((unsigned long long)sad_p[b] >> 32);
      slot2h[2 * b + 1] = (int)((unsigned long long)sad_p[b] & 0xffffffffull);
    }
    // list starts (the saddle out-crossings) and their ends, lengths, minima
    const int nch = 2 * nsb;
    std::vector<int> cstart(slot2h), q(6 * (size_t)nch);
    int *d_idx = ar2.get<int>(nch), *d_out = ar2.get<int>(6LL * nch);
    if (ar2.failed) return CASL_ENOMEM;
    CASL_CUDA_TRY(cudaMemcpyAsync(d_idx, cstart.data(), nch * sizeof(int), cudaMemcpyHostToDevice, st));
    CASL_K(k_ch_query, gsz(nch), 256, 0, st)(d_idx, nch, ta.own, jA, lA, ta.chain, ta.clev, d_out);
    RC_TRY(read_back(h, {{q.data(), d_out, q.size() * sizeof(int)}}));
    const int *cend = &q[0], *clen = &q[nch], *cmin = &q[2 * (size_t)nch],
              *val_at_min = &q[3 * (size_t)nch], *clev = &q[4 * (size_t)nch],
              *clast = &q[5 * (size_t)nch];
    std::vector<std::pair<int, int>> start2ch;
    for (int ch = 0; ch < nch; ch++) start2ch.push_back({cstart[ch], ch});
    std::sort(start2ch.begin(), start2ch.end());
    auto chain_starting_at = [&](int s) -> int {
      auto it = std::lower_bound(start2ch.begin(), start2ch.end(), std::make_pair(s, -1));
      return (it != start2ch.end() && it->first == s) ? it->second : -1;
    };
    // saddle box entered by each list's end
    std::vector<std::pair<int, long long>> end_slot(nends);
    for (int k = 0; k < nends; k++) end_slot[k] = {eidx[k], eslot[k]};
    std::sort(end_slot.begin(), end_slot.end());
    std::vector<int> box_of_end(nch);
    for (int ch = 0; ch < nch; ch++) {
      auto it = std::lower_bound(end_slot.begin(), end_slot.end(), std::make_pair(cend[ch], -1LL));
      if (it == end_slot.end() || it->first != cend[ch]) return CASL_EINVAL;
      box_of_end[ch] = (int)(std::lower_bound(sad_p.begin(), sad_p.end(), it->second) - sad_p.begin());
    }
    std::vector<int> noc(nsb, 2);
    std::vector<char> used(nch, 0);
    std::vector<int> ladd(nch, 0), lslot(nch, -1);
    std::vector<unsigned long long> skey;
    std::vector<int> sslot, sad_len;
    // lists in order of their smallest crossing: contour starts
    std::vector<int> order(nch);
    for (int k = 0; k < nch; k++) order[k] = k;
    std::sort(order.begin(), order.end(), [&](int a, int b) { return cmin[a] < cmin[b]; });
    for (int oc : order) {
      if (used[oc]) continue;
      const int icr = cmin[oc];      // the contour's first crossing
      std::vector<int> seq;          // lists in traversal order
      int ch = oc;
      used[ch] = 1;
      seq.push_back(ch);
      int guard = 0;
      while (true) {
        const int b = box_of_end[ch];
        const int k = noc[b];
        if (k < 1 || k > 2) return CASL_EINVAL;
        const int icrn = slot2h[2 * b + k - 1];
        if (icrn == icr) break;      // closes at the start (no decrement)
        noc[b] = k - 1;
        const int nxt = chain_starting_at(icrn);
        if (nxt < 0) return CASL_EINVAL;
        if (nxt == oc) break;        // back into the first list, which holds icr
        if (used[nxt]) return CASL_EINVAL;
        used[nxt] = 1;
        seq.push_back(nxt);
        ch = nxt;
        if (++guard > nch + 2) return CASL_EINVAL;
      }
      // lay out: first list rotated to start at icr, its head wrapping to the
      // end of the contour, then the others
      int L = 0;
      for (int x : seq) L += clen[x];
      const int at = C0 + nsad_contours++;
      skey.push_back((unsigned long long)(unsigned)clev[oc] << 32 | (unsigned)icr);
      sslot.push_back(at);
      sad_len.push_back(L);
      const int rot = clen[oc] - val_at_min[oc];  // place of icr in its list
      ladd[oc] = clen[oc] - rot;
      lslot[oc] = at;
      int off = clen[oc] - rot;      // crossings from icr to the list's end
      for (size_t x = 1; x < seq.size(); x++) {
        ladd[seq[x]] = clen[seq[x]] + off;
        lslot[seq[x]] = at;
        off += clen[seq[x]];
      }
    }
    for (int ch = 0; ch < nch; ch++)
      if (lslot[ch] < 0) return CASL_EINVAL;
    listof = ar2.get<int>(S);
    int *d_last = ar2.get<int>(nch);
    d_ladd = ar2.get<int>(nch);
    d_lslot = ar2.get<int>(nch);
    if (ar2.failed || C0 + nsad_contours > ccap) return CASL_ENOMEM;
    CASL_CUDA_TRY(cudaMemsetAsync(listof, 0xff, (size_t)S * sizeof(int), st));
    CASL_CUDA_TRY(cudaMemcpyAsync(d_last, clast, nch * sizeof(int), cudaMemcpyHostToDevice, st));
    CASL_CUDA_TRY(cudaMemcpyAsync(d_ladd, ladd.data(), nch * sizeof(int), cudaMemcpyHostToDevice, st));
    CASL_CUDA_TRY(cudaMemcpyAsync(d_lslot, lslot.data(), nch * sizeof(int), cudaMemcpyHostToDevice, st));
    CASL_CUDA_TRY(cudaMemcpyAsync(key + C0, skey.data(), nsad_contours * sizeof(skey[0]), cudaMemcpyHostToDevice, st));
    CASL_CUDA_TRY(cudaMemcpyAsync(slot + C0, sslot.data(), nsad_contours * sizeof(int), cudaMemcpyHostToDevice, st));
    CASL_CUDA_TRY(cudaMemcpyAsync(slen + C0, sad_len.data(), nsad_contours * sizeof(int), cudaMemcpyHostToDevice, st));
    CASL_K(k_list_of, gsz(nch), 256, 0, st)(d_last, nch, listof);
    // the host vectors must outlive their copies
    CASL_CUDA_TRY(cudaStreamSynchronize(st));
  }
  tr.point("saddles");
  // --- 7. contour order and walk layout ---------------------------------------
  const int C = C0 + nsad_contours;
  if (C == 0) return set_empty();
  {
    int lb = 1;
    while ((1 << lb) <= li.levend) lb++;
    size_t sort_bytes = 0;
    cub::DeviceRadixSort::SortPairs(nullptr, sort_bytes, key, key2, slot, slot2, C, 0, 32 + lb, st);
    void *sort_tmp = ar2.get<char>(sort_bytes + 16);
    if (ar2.failed) return CASL_ENOMEM;
    CASL_CUDA_TRY(cub::DeviceRadixSort::SortPairs(sort_tmp, sort_bytes, key, key2, slot, slot2, C, 0,
                                                  32 + lb, st));
  }
  int *clen = ar2.get<int>(C), *coff = ar2.get<int>(C), *clevt = ar2.get<int>(C), *place = ar2.get<int>(C);
  int *tmpi2 = ar2.get<int>(scan_tmp_elems(C) + 4);
  int4 *R = ar2.get<int4>(S);
  double *xw = ar2.get<double>(ncr), *yw = ar2.get<double>(ncr);
  int *cidw = ar2.get<int>(ncr);
  if (ar2.failed) return CASL_ENOMEM;
  CASL_K(k_ct_order, gsz(C), 256, 0, st)(key2, slot2, slen, C, h->p.nlevm, clen, clevt, place);
  exclusive_scan<int>(st, clen, coff, C, tmpi2, dtot + 5);
  CASL_K(k_ch_place, gsS, 256, 0, st)(head, jA, lA, ta.own, cslot, place, coff, clen, listof, d_ladd,
                                      d_lslot, S, R);
  const PlArgs pl{cg, li, uf, eg, c, coffs, ta.own, R, xw, yw, cidw};
  if (econ)
    CASL_K(k_tr_place<true>, dim3(ntile, nslice), TR_NT, 0, st)(pl);
  else
    CASL_K(k_tr_place<false>, dim3(ntile, nslice), TR_NT, 0, st)(pl);
  RC_TRY(check_launch(h));

  tr.point("layout");
  RenodeIn cur{xw, yw, coff, clen, clevt, C, ncr, nullptr, cidw};
  if (econ) {
    // one periodic image of each contour, y folded (econgen.f90:238-252)
    int *flags = ar2.get<int>(C), *klen = ar2.get<int>(C), *kone = ar2.get<int>(C);
    int *koff = ar2.get<int>(C), *kidx = ar2.get<int>(C);
    int *cs2 = ar2.get<int>(C), *len2 = ar2.get<int>(C), *lev2 = ar2.get<int>(C);
    double *xw2 = ar2.get<double>(ncr), *yw2 = ar2.get<double>(ncr);
    int *cidw2 = ar2.get<int>(ncr);
    if (ar2.failed) return CASL_ENOMEM;
    CASL_CUDA_TRY(cudaMemsetAsync(flags, 0, (size_t)C * sizeof(int), st));
    CASL_K(k_ec_flags, gsz(ncr), 256, 0, st)(yw, cidw, ncr, c, flags);
    CASL_K(k_ec_keep, gsz(C), 256, 0, st)(flags, clen, C, klen, kone);
    exclusive_scan<int>(st, klen, koff, C, tmpi2, dtot + 6);
    exclusive_scan<int>(st, kone, kidx, C, tmpi2, dtot + 7);
    int kc[2] = {0, 0};
    RC_TRY(read_back(h, {{kc, dtot + 6, 2 * sizeof(int)}}));
    if (kc[1] == 0) return set_empty();
    const double yoff = c.hly + c.elly * (double)eg.nby;
    CASL_K(k_ec_compact, gsz(ncr), 256, 0, st)(xw, yw, cidw, ncr, coff, klen, koff, kidx, c, yoff, xw2,
                                        yw2, cidw2);
    CASL_K(k_ec_contours, gsz(C), 256, 0, st)(clen, clevt, C, klen, koff, kidx, cs2, len2, lev2);
    RC_TRY(check_launch(h));
    cur = RenodeIn{xw2, yw2, cs2, len2, lev2, kc[1], kc[0], nullptr, cidw2};
    tr.point("one image");
  }
  // --- 8. renode three times (congen.f90:295-310) -----------------------------
  long long capn = std::max<long long>(ncr * 2, h->npm);
  double *xa = ar2.get<double>(capn), *ya = ar2.get<double>(capn);
  double *xb = ar2.get<double>(capn), *yb = ar2.get<double>(capn);
  int *ocs[2], *olen[2], *olev[2];
  for (int q = 0; q < 2; q++) {
    ocs[q] = ar2.get<int>(C); olen[q] = ar2.get<int>(C); olev[q] = ar2.get<int>(C);
  }
  int *cnt = ar2.get<int>(4);
  if (ar2.failed) return CASL_ENOMEM;
  double *ox[3] = {xa, xb, xa}, *oy[3] = {ya, yb, ya};
  int hc[3] = {0, 0, 0};
  for (int pass = 0; pass < 3; pass++) {
    RenodeOut out{};
    out.xo = ox[pass]; out.yo = oy[pass];
    out.ocs = ocs[pass & 1]; out.olen = olen[pass & 1]; out.olev = olev[pass & 1];
    out.cap = capn;
    out.d_counts = cnt;
    size_t mark = ar2.off;
    RC_TRY(renode_batch(h, ar2, cur, out, RENODE_PLAIN));
    ar2.off = mark;
    RC_TRY(read_back(h, {{hc, cnt, 3 * sizeof(int)}}));
    if (hc[2]) return CASL_ECAPACITY;
    if (hc[0] == 0) return set_empty();
    cur = RenodeIn{out.xo, out.yo, out.ocs, out.olen, out.olev, hc[0], hc[1]};
    tr.point(pass == 0 ? "renode1" : (pass == 1 ? "renode2" : "renode3"));
  }
  int nq = hc[0], npt = hc[1];
  if (npt > h->npm || nq > h->nm) return CASL_ECAPACITY;
  CASL_CUDA_TRY(cudaMemcpyAsync(h->xq, cur.xw, (size_t)npt * sizeof(double), cudaMemcpyDeviceToDevice, st));
  CASL_CUDA_TRY(cudaMemcpyAsync(h->yq, cur.yw, (size_t)npt * sizeof(double), cudaMemcpyDeviceToDevice, st));
  CASL_K(k_out_contours, gsz(nq), 256, 0, st)(cur.cs, cur.len, cur.levt, nq, h->i1q, h->i2q, h->npq,
                                          h->indq);
  CASL_K(k_out_links, gsz(npt), 256, 0, st)(cur.cs, cur.len, nq, npt, h->nextq);
  CASL_K(k_set_counts2, 1, 1, 0, st)(h->scal, cnt);
  RC_TRY(check_launch(h));
  h->nq = nq;
  h->nptq = npt;
  h->contex = npt > 0;
  return CASL_OK;
}

}  // namespace casl

// ---------------------------------------------------------------------------
// genfg (post/genfg.f90:79-194): the PV on the ultra-fine grid as an image
// ---------------------------------------------------------------------------
namespace casl {

// out(iy, ix) = real(qa(iy1 + iy*stride, ix1 + ix*stride)), periodic, 0-based
// starts, out column-major (nyv, nxv)
__global__ void k_gf_gather(const double *__restrict__ qa, int nxu, int nyu, int ix1, int nxv,
                            int iy1, int nyv, int stride, float *__restrict__ out) {
  CASL_PDL_ENTRY();
  const long long m = (long long)nxv * nyv;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < m;
       t += (long long)gridDim.x * blockDim.x) {
    int iy = (int)(t % nyv), ix = (int)(t / nyv);
    long long sx = ((long long)ix1 + (long long)ix * stride) % nxu;
    long long sy = ((long long)iy1 + (long long)iy * stride) % nyu;
    out[t] = (float)qa[sx * nyu + sy];
  }
}

}  // namespace casl

using namespace casl;

extern "C" int casl_genfg(casl_handle *h, int ix1v, int nxv, int iy1v, int nyv, int stride,
                          float *out) {
  if (!h || !out) return CASL_EINVAL;
  if (h->M > 1) return CASL_EUNSUPPORTED;  // one simulation's image
  const Consts &c = h->c;
  const int nxu = c.nxu, nyu = c.nyu;
  if (ix1v < 1 || ix1v > nxu || iy1v < 1 || iy1v > nyu || nxv < 1 || nyv < 1 || stride < 1 ||
      (long long)(nxv - 1) * stride >= nxu || (long long)(nyv - 1) * stride >= nyu)
    return CASL_EINVAL;
  int rc = sync_counts(h);
  if (rc) return rc;
  cudaStream_t st = h->stream;
  const long long NU = (long long)nxu * nyu, m = (long long)nxv * nyv;
  size_t need = (size_t)NU * 12 + (size_t)nxu * 4 + (size_t)m * 4 + ((size_t)64 << 20);
  RC_TRY(ensure_scratch(h, need));
  Arena ar{(char *)h->sx, h->sx_bytes, 0};
  double *qa = ar.get<double>(NU);
  int *Lu = ar.get<int>(NU);
  int *ljx = ar.get<int>(nxu);
  unsigned long long *lsum = ar.get<unsigned long long>(4);
  float *img = ar.get<float>(m);
  if (ar.failed) return CASL_ENOMEM;
  // con2ugrid (congen.f90:338-441), always called by genfg, then the
  // bilinear residual qr (genfg.f90:95-109)
  CASL_CUDA_TRY(cudaMemsetAsync(Lu, 0, (size_t)NU * sizeof(int), st));
  CASL_CUDA_TRY(cudaMemsetAsync(ljx, 0, (size_t)nxu * sizeof(int), st));
  CASL_CUDA_TRY(cudaMemsetAsync(lsum, 0, 4 * sizeof(unsigned long long), st));
  if (h->nptq > 0)
    CASL_K(k_u_scatter, gsz(h->nptq), 256, 0, st)(h->xq, h->yq, h->nextq, h->nptq, h->qjump, Lu,
                                              ljx, c, &h->scal->error);
  CASL_K(k_u_lbot, 1, 1024, 0, st)(ljx, Lu, nxu, nyu);
  CASL_K(k_u_colscan, (nxu * 32 + 255) / 256, 256, 0, st)(Lu, nxu, nyu, lsum);
  LevInfo lq{0, 0, h->qjump, 0.0, 1.0};
  CASL_K(k_u_field, 4096, 256, 0, st)(Lu, lsum, h->qr, h->qjump, 1, lq, qa, nullptr, lsum + 1, c, 0.0);
  CASL_K(k_gf_gather, gsz(m), 256, 0, st)(qa, nxu, nyu, ix1v - 1, nxv, iy1v - 1, nyv, stride, img);
  RC_TRY(check_launch(h));
  CASL_CUDA_TRY(cudaMemcpyAsync(out, img, (size_t)m * sizeof(float), cudaMemcpyDeviceToHost, st));
  return read_back(h, {});
}

// The spectral work of one RK4 stage (evolution.f90:166-326) in four launches:
//
//   k_fs_cols   con2grid's forward transform along iy            (column CTAs)
//   k_fs_rows   its transform along ix, the filter combination that forms qq
//               and pp (evolution.f90:507-514), and the kx half of the inverse
//               transforms of u, v and the four gradients            (row CTAs)
//   k_fs_prod   their ky half, the advection products and the iy half of the
//               products' forward transforms                     (column CTAs)
//   k_fs_end    the ix half, damping and integrating factor, the RK4 update of
//               qs and qd -- and, in further blocks, the node update  (row CTAs)
//
// A 2-D transform needs all rows before any column, so these are as many
// passes as the chain of transforms has axis changes; everything pointwise
// between two changes happens in the CTA that already holds the row or column.
// Against one launch per transform and axis plus elementwise kernels between
// them, the four gradients and the products' inputs never reach memory, the
// intermediates of u, v and the gradients are written and read once, and a
// stage takes 4 launches for 7 (8 in stage 1, whose vorticity transform for
// adapt joins k_fs_rows and k_fs_prod).
//
// Measured at 1024^2, 1.4M nodes (B200): the transforms, combination, factors
// and updates of a step took 940 us as separate launches and take 718 us
// (k_fs_cols 59, k_fs_rows 196, k_fs_prod 210, k_fs_end 110, nodes 143).  At
// 64^2, where a launch costs its latency, a step went from 360 to 275 us.
// k_fs_rows and k_fs_prod are bound by shared-memory wavefronts (60 % of the
// cycles at 1024^2: the exchanges of the transforms), with the FP64 pipe 28 %
// busy and DRAM 13 %; k_fs_end and the nodes by memory latency.
//
// Two real vectors per complex transform.  Every pass packs two adjacent
// vectors a, b of the same field as z = a + ib, so a length-n complex
// transform carries both and the even/odd untangling of a real transform
// becomes one pairing of z(k) with z(n-k).  Vectors of one field are of one
// size, so neither picks up the other's rounding.
//
// Layouts.  What a row CTA writes for column CTAs is stored in tiles of four
// columns, tile (ix/4): [ky][ix%4], so that a column CTA's input is one
// contiguous run per field, staged by one bulk copy; the row CTA's stores are
// whole 32-byte sectors.  What a column CTA writes for row CTAs is [ky][ix],
// four columns (one sector) per row.
#pragma once

#include "fft.cuh"
#include "state.cuh"

namespace casl {

// Complex transform of length N = 2^LOGN, x holding Z[t + m*TPV] before and
// after (TPV = N/8); at(i) is the thread's transform's exchange slot element
// i, sync() joins the transform's threads.
template <int LOGN, bool FWD, class At, class Sync>
__device__ __forceinline__ void cfft(double2 (&x)[8], int t, const double2 *__restrict__ tw, At at,
                                     Sync sync) {
  constexpr int N = 1 << LOGN, TPV = N / 8, P8 = LOGN / 3, REM = LOGN % 3;
  int Ns = 1;
#pragma unroll
  for (int p = 0; p < P8; p++) {
    rf_butterflies<8, FWD, TPV>(x, t, Ns, tw, N);
    if (p < P8 - 1 || REM != 0) {
      const int base = (t / Ns) * Ns * 8 + (t & (Ns - 1));
#pragma unroll
      for (int r = 0; r < 8; r++) at(base + r * Ns) = x[r];
      sync();
#pragma unroll
      for (int m = 0; m < 8; m++) x[m] = at(t + m * TPV);
      sync();
    }
    Ns *= 8;
  }
  if (REM == 2) rf_butterflies<4, FWD, TPV>(x, t, Ns, tw, N);
  if (REM == 1) rf_butterflies<2, FWD, TPV>(x, t, Ns, tw, N);
}

// Joins the TPV threads of transform g of a block: inside a warp, or a named
// barrier (ids 1..15) where a transform spans several.
template <int TPV>
__device__ __forceinline__ void group_sync(int g) {
  if constexpr (TPV >= 64) {
    asm volatile("bar.sync %0, %1;" ::"r"(g + 1), "n"(TPV) : "memory");
  } else if constexpr (TPV == 32) {
    __syncwarp();
  } else {
    __syncwarp(((1u << TPV) - 1u) << ((threadIdx.x & 31) & ~(TPV - 1)));
  }
}

// The exchange slot of a length-N transform: one spare element per eight.
template <int LOGN>
constexpr int fs_slot() { return (1 << LOGN) + (1 << LOGN) / 8; }

// z(k), z(n-k) of a forward transform of a + ib -> rows k and n-k of the
// Hermitian layout, as (a, b) pairs.
__device__ __forceinline__ void fs_untangle(double2 zk, double2 zc, double s, double2 &lo,
                                            double2 &hi) {
  lo = make_double2(0.5 * (zk.x + zc.x) * s, 0.5 * (zk.y + zc.y) * s);
  hi = make_double2(0.5 * (zk.y - zc.y) * s, 0.5 * (zc.x - zk.x) * s);
}
// Element kk of the packed spectrum z of two Hermitian vectors: (ar, br) and
// (ai, bi) are their elements k and n-k, k = min(kk, n-kk), 0 < k < n/2.
__device__ __forceinline__ double2 fs_tangle(bool hi, double ar, double ai, double br, double bi) {
  return hi ? make_double2(ar + bi, br - ai) : make_double2(ar - bi, ai + br);
}

__device__ __forceinline__ void st2(double *p, double a, double b) {
  *reinterpret_cast<double2 *>(p) = make_double2(a, b);
}

// ---------------------------------------------------------------------------
// con2grid's forward transform along iy
// ---------------------------------------------------------------------------
// Four columns (two packed transforms, interleaved over the lanes) per tile.
// The blocks past `ncol` clear the packed jump words that con2grid's sum has
// finished with, for the next stage's scatter: this launch has one field's
// worth of transforms (256 CTAs at n = 1024) and leaves the memory idle,
// where a clear of its own took 9.6 us (33 MB, n = 1024) and a launch.
template <int LOGN>
struct FsCols {
  static constexpr int N = 1 << LOGN, TPV = N / 8, GT = 2 * TPV;
  static constexpr int TPC = GT >= 32 ? 1 : 32 / GT;  // tiles per CTA
  static constexpr int NT = GT * TPC;
  static constexpr size_t smem = (size_t)TPC * 2 * fs_slot<LOGN>() * sizeof(double2);
};
struct ClearJob {
  uint4 *words;       // the packed jumps, 16-byte units
  long long nwords;
  int *ljx;
  long long nljx;
};
template <int LOGN>
__global__ void __launch_bounds__(FsCols<LOGN>::NT, (1024 / FsCols<LOGN>::NT > 16 ? 16 : 1024 / FsCols<LOGN>::NT))
    k_fs_cols(LoadQC ld, double *__restrict__ T, const double2 *__restrict__ tw, int ncol,
              ClearJob clr) {
  CASL_PDL_ENTRY();
  using Sh = FsCols<LOGN>;
  constexpr int N = Sh::N, TPV = Sh::TPV, SL = fs_slot<LOGN>();
  if ((int)blockIdx.x >= ncol) {
    const long long nb = (long long)(gridDim.x - ncol) * gridDim.y;
    const long long id = ((long long)blockIdx.y * (gridDim.x - ncol) + blockIdx.x - ncol) * Sh::NT + threadIdx.x;
    const long long stride = nb * Sh::NT;
    for (long long i = id; i < clr.nwords; i += stride) clr.words[i] = make_uint4(0, 0, 0, 0);
    for (long long i = id; i < clr.nljx; i += stride) clr.ljx[i] = 0;
    return;
  }
  extern __shared__ double2 smem[];
  const int tile = threadIdx.x / Sh::GT, lt = threadIdx.x - tile * Sh::GT;
  const int g = lt & 1, t = lt >> 1, b = blockIdx.y;
  const int ix = ((int)blockIdx.x * Sh::TPC + tile) * 4 + 2 * g;
  double2 *S = smem + tile * 2 * SL;
  auto at = [&](int i) -> double2 & { return S[cpad(i) * 2 + g]; };
  auto sync = [] { __syncthreads(); };
  double2 x[8];
#pragma unroll
  for (int m = 0; m < 8; m++) {
    const int j = t + m * TPV;
    x[m] = make_double2(ld(b, ix, j), ld(b, ix + 1, j));
  }
  cfft<LOGN, true>(x, t, tw, at, sync);
#pragma unroll
  for (int m = 0; m < 8; m++) at(t + m * TPV) = x[m];
  __syncthreads();
  const double s = 1.0 / sqrt((double)N);
  double *o = T + (long long)b * N * N + ix;
#pragma unroll
  for (int m = 0; m < 4; m++) {
    const int k = t + m * TPV;
    if (k == 0) {
      const double2 z0 = at(0), zh = at(N / 2);
      st2(o, z0.x * s, z0.y * s);
      st2(o + (N / 2) * N, zh.x * s, zh.y * s);
    } else {
      double2 lo, hi;
      fs_untangle(at(k), at(N - k), s, lo, hi);
      st2(o + k * N, lo.x, lo.y);
      st2(o + (N - k) * N, hi.x, hi.y);
    }
  }
}

// ---------------------------------------------------------------------------
// Rows: forward along ix, filter combination, inverse along kx
// ---------------------------------------------------------------------------
// A pair of rows (ky, ky+1) per three transforms' threads: the forward
// transform of con2grid's rows packs the pair, then the three groups take pp
// (for v and u), qd and qs, each an x derivative and a y derivative of the
// packed pair.  Rows of con2grid's spectrum, qd and qs arrive by bulk copies.
template <int LOGN>
struct FsRows {
  static constexpr int N = 1 << LOGN, TPV = N / 8, GPT = 3 * TPV;
  static constexpr int P = GPT >= 96 ? 1 : 96 / GPT;  // row pairs per CTA
  static constexpr int NT = GPT * P;
  static constexpr size_t rows = (size_t)P * 6 * N * sizeof(double);
  static constexpr size_t smem = rows + (size_t)P * 3 * fs_slot<LOGN>() * sizeof(double2) + 16;
  static constexpr int MINB = LOGN >= 11 ? 1 : (LOGN >= 9 ? 2 : 4);
};
struct FsRowArgs {
  const double *tqc;             // con2grid's half-transformed field [ky][ix]
  double *qs, *qd, *qc, *qq, *pp;
  const double *flo, *fhi, *green, *hrkx, *hrky;
  double *t6;                    // six fields, tiled
  double *tzz;                   // stage 1: the vorticity's half-transform, tiled
  double kdsq;
  int btropic;
  int have;                      // contours exist (else qc = 0)
  int keep;                      // write qc, qq and pp
  int *err;
};
template <int LOGN, bool FIRST>
__global__ void __launch_bounds__(FsRows<LOGN>::NT, FsRows<LOGN>::MINB)
    k_fs_rows(FsRowArgs a, const double2 *__restrict__ tw) {
  CASL_PDL_ENTRY();
  using Sh = FsRows<LOGN>;
  constexpr int N = Sh::N, TPV = Sh::TPV, P = Sh::P, NT = Sh::NT, SL = fs_slot<LOGN>();
  constexpr long long nn = (long long)N * N;
  extern __shared__ double2 smem[];
  double *R = reinterpret_cast<double *>(smem);  // per pair: A, D, Q of 2N
  double2 *slots = smem + Sh::rows / sizeof(double2);
  uint64_t *bar = reinterpret_cast<uint64_t *>(slots + P * 3 * SL);
  const long long mo = blockIdx.y * nn;  // ensemble member
  const int pair0 = blockIdx.x * P;
  if (threadIdx.x == 0) {
    tc::mbar_init(bar, 1);
    tc::mbar_fence_init();
    tc::mbar_expect_tx(bar, (uint32_t)(P * (a.have ? 3 : 2) * 2 * N * 8));
#pragma unroll 1
    for (int p = 0; p < P; p++) {
      const long long o = mo + (long long)(pair0 + p) * 2 * N;
      double *d = R + p * 6 * N;
      if (a.have) tc::bulk_g2s(d, a.tqc + o, 2 * N * 8, bar);
      tc::bulk_g2s(d + 2 * N, a.qd + o, 2 * N * 8, bar);
      tc::bulk_g2s(d + 4 * N, a.qs + o, 2 * N * 8, bar);
    }
  }
  __syncthreads();
  if (!tc::mbar_wait(bar, 0) && threadIdx.x == 0) atomicExch(a.err, CASL_ETIMEOUT);
  const int grp = threadIdx.x / TPV, t = threadIdx.x - grp * TPV;
  const int lp = grp / 3, f = grp - lp * 3;
  const int r0 = 2 * (pair0 + lp);
  double *A = R + lp * 6 * N;
  double2 *S = slots + grp * SL;
  auto at = [&](int i) -> double2 & { return S[cpad(i)]; };
  auto sync = [&] { group_sync<TPV>(grp); };
  const double s = 1.0 / sqrt((double)N);
  double2 x[8];
  if (f == 0 && a.have) {
#pragma unroll
    for (int m = 0; m < 8; m++) {
      const int j = t + m * TPV;
      x[m] = make_double2(A[j], A[N + j]);
    }
    cfft<LOGN, true>(x, t, tw, at, sync);
#pragma unroll
    for (int m = 0; m < 8; m++) at(t + m * TPV) = x[m];
    sync();
#pragma unroll
    for (int m = 0; m < 4; m++) {
      const int k = t + m * TPV;
      if (k == 0) {
        const double2 z0 = at(0), zh = at(N / 2);
        A[0] = z0.x * s;
        A[N] = z0.y * s;
        A[N / 2] = zh.x * s;
        A[N + N / 2] = zh.y * s;
      } else {
        double2 lo, hi;
        fs_untangle(at(k), at(N - k), s, lo, hi);
        A[k] = lo.x;
        A[N + k] = lo.y;
        A[N - k] = hi.x;
        A[N + N - k] = hi.y;
      }
    }
  }
  __syncthreads();
  // qq = flo*(qs-qc)+qc+qd, pp = green*qq; stage 1 also resets qs <- qq,
  // qd <- fhi*(qs-qc) (evolution.f90:199-200).  pp takes qc's place.
  for (int e = threadIdx.x; e < P * N; e += NT) {
    const int p = e >> LOGN, k = 2 * (e & (N - 1));
    double *B = R + p * 6 * N + k;
    const long long kt = (long long)(pair0 + p) * 2 * N + k, o = mo + kt;
    const double2 fl = __ldg(reinterpret_cast<const double2 *>(a.flo + kt));
    const double2 gr = __ldg(reinterpret_cast<const double2 *>(a.green + kt));
    double2 c = make_double2(0.0, 0.0);
    if (a.have) c = *reinterpret_cast<double2 *>(B);
    const double2 d = *reinterpret_cast<double2 *>(B + 2 * N);
    const double2 q = *reinterpret_cast<double2 *>(B + 4 * N);
    const double q0 = fl.x * (q.x - c.x) + c.x + d.x, q1 = fl.y * (q.y - c.y) + c.y + d.y;
    const double p0 = gr.x * q0, p1 = gr.y * q1;
    st2(B, p0, p1);
    if (a.keep) {
      st2(a.qc + o, c.x, c.y);
      st2(a.qq + o, q0, q1);
      st2(a.pp + o, p0, p1);
    }
    if (FIRST) {
      const double2 fh = __ldg(reinterpret_cast<const double2 *>(a.fhi + kt));
      const double d0 = fh.x * (q0 - c.x), d1 = fh.y * (q1 - c.y);
      st2(B + 4 * N, q0, q1);
      st2(B + 2 * N, d0, d1);
      st2(a.qs + o, q0, q1);
      st2(a.qd + o, d0, d1);
    }
  }
  __syncthreads();
  const double *F0 = A + (f == 0 ? 0 : 2 * N * f), *F1 = F0 + N;  // pp, qd, qs
  double *out = a.t6 + (blockIdx.y * 6 + 2 * f) * nn;
  auto put = [&](double *dst, int ra, int rb) {
#pragma unroll
    for (int m = 0; m < 8; m++) {
      const int j = t + m * TPV;
      const long long o = (long long)(j >> 2) * (4 * N) + (j & 3);
      dst[o + ra * 4] = x[m].x * s;
      dst[o + rb * 4] = x[m].y * s;
    }
  };
  // x derivative (sta2dfft.f90:169-204): element k takes -h times element
  // n-k, element n-k h times element k; 0 at k = 0, n/2
#pragma unroll
  for (int m = 0; m < 8; m++) {
    const int kk = t + m * TPV;
    if (kk == 0 || kk == N / 2) {
      x[m] = make_double2(0.0, 0.0);
    } else {
      const bool hi = kk > N / 2;
      const int k = hi ? N - kk : kk;
      const double h = __ldg(&a.hrkx[2 * k - 1]);
      x[m] = fs_tangle(hi, -h * F0[N - k], h * F0[k], -h * F1[N - k], h * F1[k]);
    }
  }
  cfft<LOGN, false>(x, t, tw, at, sync);
  put(out, r0, r0 + 1);
  // y derivative: row j of it is a factor of row n-j, so rows r0, r0+1 give
  // rows n-r0, n-r0-1
  auto yfac = [&](int j) {
    if (j == 0 || j == N / 2) return 0.0;
    return j < N / 2 ? -__ldg(&a.hrky[2 * j - 1]) : __ldg(&a.hrky[2 * (N - j) - 1]);
  };
  const int ja = (N - r0) & (N - 1), jb = N - r0 - 1;
  const double fa = yfac(ja), fb = yfac(jb);
#pragma unroll
  for (int m = 0; m < 8; m++) {
    const int kk = t + m * TPV;
    if (kk == 0 || kk == N / 2) {
      x[m] = make_double2(fa * F0[kk], fb * F1[kk]);
    } else {
      const bool hi = kk > N / 2;
      const int k = hi ? N - kk : kk;
      x[m] = fs_tangle(hi, fa * F0[k], fa * F0[N - k], fb * F1[k], fb * F1[N - k]);
    }
  }
  cfft<LOGN, false>(x, t, tw, at, sync);
  put(out + nn, ja, jb);
  if (FIRST && f == 0) {
    // qq + kdsq*pp (evolution.f90:541-547), qq as this block has just written it
    const double *Q0 = a.qq + mo + (long long)r0 * N;
    auto V = [&](int r, int k) {
      const double q = Q0[r * N + k];
      return a.btropic ? q : q + a.kdsq * F0[r * N + k];
    };
#pragma unroll
    for (int m = 0; m < 8; m++) {
      const int kk = t + m * TPV;
      if (kk == 0 || kk == N / 2) {
        x[m] = make_double2(V(0, kk), V(1, kk));
      } else {
        const bool hi = kk > N / 2;
        const int k = hi ? N - kk : kk;
        x[m] = fs_tangle(hi, V(0, k), V(0, N - k), V(1, k), V(1, N - k));
      }
    }
    cfft<LOGN, false>(x, t, tw, at, sync);
    put(a.tzz + mo, r0, r0 + 1);
  }
}

// ---------------------------------------------------------------------------
// Columns: inverse along ky, advection products, forward along iy
// ---------------------------------------------------------------------------
// Four columns per tile, four transforms interleaved over the lanes: lane
// g = 2p + q takes columns 2p, 2p+1 of field q of a pair (v and u, then the
// x and y derivatives of qd, then of qs), and one shuffle per value hands
// each lane both fields of its own column, 2p + q.  The products are packed
// by columns again, the even lanes taking qd's and the odd lanes qs's.  The
// tile's input is staged over the exchange slots, which are written only
// after it has been read.
template <int LOGN>
struct FsProd {
  static constexpr int N = 1 << LOGN, TPV = N / 8, GT = 4 * TPV;
  static constexpr int TPC = GT >= 32 ? 1 : 32 / GT;  // tiles per CTA
  static constexpr int NT = GT * TPC;
  static constexpr size_t slots = (size_t)TPC * 4 * fs_slot<LOGN>() * sizeof(double2);
  static constexpr size_t smem = slots + (size_t)NT * 8 * sizeof(double) + 16;
  static constexpr int MINB = 1024 / NT > 8 ? 8 : 1024 / NT;
};
struct FsProdArgs {
  const double *t6;
  const double *tzz;
  double *uu, *vv;       // physical [ix][iy]
  double *tp;            // the two products' half-transforms [ky][ix]
  double *part;          // stage 1: block sums and maxima for adapt
  double betab;
  int *err;
};
template <int LOGN, bool FIRST>
__global__ void __launch_bounds__(FsProd<LOGN>::NT, FsProd<LOGN>::MINB)
    k_fs_prod(FsProdArgs a, const double2 *__restrict__ tw) {
  CASL_PDL_ENTRY();
  using Sh = FsProd<LOGN>;
  constexpr int N = Sh::N, TPV = Sh::TPV, TPC = Sh::TPC, NT = Sh::NT, SL = fs_slot<LOGN>();
  constexpr long long nn = (long long)N * N;
  extern __shared__ double2 smem[];
  double *stash = reinterpret_cast<double *>(smem + TPC * 4 * SL) + threadIdx.x;
  uint64_t *bar = reinterpret_cast<uint64_t *>(reinterpret_cast<double *>(smem + TPC * 4 * SL) + NT * 8);
  const int tile = threadIdx.x / Sh::GT, lt = threadIdx.x - tile * Sh::GT;
  const int g = lt & 3, t = lt >> 2, p = g >> 1, q = g & 1;
  const int blk0 = blockIdx.x * TPC, ix0 = (blk0 + tile) * 4;
  double2 *S = smem + tile * 4 * SL;
  auto at = [&](int i) -> double2 & { return S[cpad(i) * 4 + g]; };
  auto sync = [] { __syncthreads(); };
  const double s = 1.0 / sqrt((double)N);
  if (threadIdx.x == 0) {
    tc::mbar_init(bar, 1);
    tc::mbar_fence_init();
  }
  // field q of the staged pair begins 64 bytes past a bank period, so that
  // the even and odd lanes' reads do not meet
  constexpr int FO = 4 * N + 8;
  const double *t6 = a.t6 + blockIdx.y * 6 * nn;
  double *ucol = a.uu + blockIdx.y * nn + (long long)(ix0 + g) * N;
  double *vcol = a.vv + blockIdx.y * nn + (long long)(ix0 + g) * N;
  const unsigned full = NT >= 32 ? 0xffffffffu : (1u << NT) - 1u;
  double umax = 0.0;
  double2 x[8];
#pragma unroll 1
  for (int fp = 0; fp < 3; fp++) {
    tc::fence_proxy_async_smem();
    __syncthreads();
    if (threadIdx.x == 0) {
      constexpr uint32_t bytes = 4 * N * 8;
      tc::mbar_expect_tx(bar, TPC * 2 * bytes);
#pragma unroll 1
      for (int c = 0; c < TPC; c++) {
        double *d = reinterpret_cast<double *>(smem + c * 4 * SL);
        const double *src = t6 + 2 * fp * nn + (long long)(blk0 + c) * 4 * N;
        tc::bulk_g2s(d, src, bytes, bar);
        tc::bulk_g2s(d + FO, src + nn, bytes, bar);
      }
    }
    if (!tc::mbar_wait(bar, fp & 1) && threadIdx.x == 0) atomicExch(a.err, CASL_ETIMEOUT);
    const double *F = reinterpret_cast<const double *>(S) + q * FO + 2 * p;
#pragma unroll
    for (int m = 0; m < 8; m++) {
      const int kk = t + m * TPV;
      if (kk == 0 || kk == N / 2) {
        x[m] = ld2(F + kk * 4);
      } else {
        const bool hi = kk > N / 2;
        const int k = hi ? N - kk : kk;
        const double2 re = ld2(F + k * 4), im = ld2(F + (N - k) * 4);
        x[m] = fs_tangle(hi, re.x, im.x, re.y, im.y);
      }
    }
    __syncthreads();
    cfft<LOGN, false>(x, t, tw, at, sync);
    // both fields of this lane's column: (d/dx, d/dy)
#pragma unroll
    for (int m = 0; m < 8; m++) {
      const double r = __shfl_xor_sync(full, q ? x[m].x : x[m].y, 1);
      x[m] = q ? make_double2(r * s, x[m].y * s) : make_double2(x[m].x * s, r * s);
    }
    if (fp == 0) {
#pragma unroll
      for (int m = 0; m < 8; m++) {
        const double v = x[m].x, u = -x[m].y;
        vcol[t + m * TPV] = v;
        ucol[t + m * TPV] = u;
        if (FIRST) umax = fmax(umax, u * u + v * v);
      }
    } else {
#pragma unroll
      for (int m = 0; m < 8; m++) {
        const double u = ucol[t + m * TPV], v = vcol[t + m * TPV];
        const double gx = x[m].x;
        double gy = x[m].y;
        if (fp == 2 && a.betab != 0.0) gy = gy + a.betab;
        const double pr = -u * gx - v * gy;
        if (fp == 1)
          stash[m * NT] = pr;
        else
          x[m].x = pr;
      }
    }
  }
  // products: the even lane of a column pair takes qd's, the odd lane qs's
#pragma unroll
  for (int m = 0; m < 8; m++) {
    const double pd = stash[m * NT], ps = x[m].x;
    const double r = __shfl_xor_sync(full, q ? pd : ps, 1);
    x[m] = q ? make_double2(r, ps) : make_double2(pd, r);
  }
  cfft<LOGN, true>(x, t, tw, at, sync);
#pragma unroll
  for (int m = 0; m < 8; m++) at(t + m * TPV) = x[m];
  __syncthreads();
  double *o = a.tp + (blockIdx.y * 2 + q) * nn + ix0 + 2 * p;
#pragma unroll
  for (int m = 0; m < 4; m++) {
    const int k = t + m * TPV;
    if (k == 0) {
      const double2 z0 = at(0), zh = at(N / 2);
      st2(o, z0.x * s, z0.y * s);
      st2(o + (N / 2) * N, zh.x * s, zh.y * s);
    } else {
      double2 lo, hi;
      fs_untangle(at(k), at(N - k), s, lo, hi);
      st2(o + k * N, lo.x, lo.y);
      st2(o + (N - k) * N, hi.x, hi.y);
    }
  }
  if (FIRST) {
    // the vorticity's columns (the even lanes'), for adapt's rms and maximum
    tc::fence_proxy_async_smem();
    __syncthreads();
    if (threadIdx.x == 0) {
      constexpr uint32_t bytes = 4 * N * 8;
      tc::mbar_expect_tx(bar, TPC * bytes);
#pragma unroll 1
      for (int c = 0; c < TPC; c++)
        tc::bulk_g2s(smem + c * 4 * SL, a.tzz + blockIdx.y * nn + (long long)(blk0 + c) * 4 * N,
                     bytes, bar);
    }
    if (!tc::mbar_wait(bar, 1) && threadIdx.x == 0) atomicExch(a.err, CASL_ETIMEOUT);
    const double *F = reinterpret_cast<const double *>(S) + 2 * p;
#pragma unroll
    for (int m = 0; m < 8; m++) {
      const int kk = t + m * TPV;
      if (q) {
        x[m] = make_double2(0.0, 0.0);
      } else if (kk == 0 || kk == N / 2) {
        x[m] = ld2(F + kk * 4);
      } else {
        const bool hi = kk > N / 2;
        const int k = hi ? N - kk : kk;
        const double2 re = ld2(F + k * 4), im = ld2(F + (N - k) * 4);
        x[m] = fs_tangle(hi, re.x, im.x, re.y, im.y);
      }
    }
    __syncthreads();
    cfft<LOGN, false>(x, t, tw, at, sync);
    double sum = 0.0, zmax = 0.0;
#pragma unroll
    for (int m = 0; m < 8; m++) {
      const double z0 = x[m].x * s, z1 = x[m].y * s;
      sum += z0 * z0 + z1 * z1;
      zmax = fmax(zmax, fmax(z0 * z0, z1 * z1));
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
      sum += __shfl_down_sync(full, sum, d);
      zmax = fmax(zmax, __shfl_down_sync(full, zmax, d));
      umax = fmax(umax, __shfl_down_sync(full, umax, d));
    }
    __syncthreads();
    double *red = reinterpret_cast<double *>(smem);
    const int wid = threadIdx.x >> 5;
    if ((threadIdx.x & 31) == 0) {
      red[3 * wid] = sum;
      red[3 * wid + 1] = zmax;
      red[3 * wid + 2] = umax;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      for (int w = 1; w < NT / 32; w++) {
        sum += red[3 * w];
        zmax = fmax(zmax, red[3 * w + 1]);
        umax = fmax(umax, red[3 * w + 2]);
      }
      double *o3 = a.part + 3 * ((long long)blockIdx.y * gridDim.x + blockIdx.x);
      o3[0] = sum;
      o3[1] = zmax;
      o3[2] = umax;
    }
  }
}

// ---------------------------------------------------------------------------
// Rows: forward along ix, source terms, RK4 update; and the node update
// ---------------------------------------------------------------------------
// A pair of rows of both products per CTA (group 0 qd's, group 1 qs's), so
// each transform's threads finish their field's RK4 update at the elements
// they hold.  The update's rows are asked into L2 while the transform runs.
template <int LOGN>
struct FsEnd {
  static constexpr int N = 1 << LOGN, TPV = N / 8, GPT = 2 * TPV;
  static constexpr int NT = GPT >= 128 ? GPT : 128;
  static constexpr int P = NT / GPT;  // row pairs per CTA
  static constexpr int ROWB = N / (2 * P) > 0 ? N / (2 * P) : 1;
  static constexpr size_t smem = (size_t)2 * P * fs_slot<LOGN>() * sizeof(double2);
};
struct FsEndArgs {
  const double *tp;
  double *qs, *qd, *qsi, *qsf, *qdi, *qdf, *emq, *epq;
  const double *qq, *pp, *qdiss;
  double rekman, kdsq, therm;
  int heating, friction;
};
__device__ __forceinline__ void l2_prefetch(const void *p, uint32_t bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}
// The qs update of a stage (evolution.f90:212-311) at four elements.  All
// loads come before the first store: the arrays may alias as far as the
// compiler knows, and one element after the other would wait for memory four
// times.
template <int STAGE>
__device__ __forceinline__ void fs_rk_qs(const FsEndArgs &a, const Scalars &sm,
                                         const long long (&i)[4], const double (&x)[4]) {
  double s0[4], sf[4];
#pragma unroll
  for (int e = 0; e < 4; e++) {
    if (STAGE == 1) s0[e] = a.qs[i[e]];
    if (STAGE == 2 || STAGE == 3) s0[e] = a.qsi[i[e]];
    if (STAGE != 1) sf[e] = a.qsf[i[e]];
  }
  const double dt = sm.dt, dt2 = sm.dt2, dt3 = sm.dt3, dt6 = sm.dt6;
#pragma unroll
  for (int e = 0; e < 4; e++) {
    if (STAGE == 1) {
      a.qsi[i[e]] = s0[e];
      a.qs[i[e]] = s0[e] + dt2 * x[e];
      a.qsf[i[e]] = s0[e] + dt6 * x[e];
    } else if (STAGE == 4) {
      a.qs[i[e]] = sf[e] + dt6 * x[e];
    } else {
      a.qs[i[e]] = s0[e] + (STAGE == 2 ? dt2 : dt) * x[e];
      a.qsf[i[e]] = sf[e] + dt3 * x[e];
    }
  }
}
// qd's source (damping and integrating factor, evolution.f90:466-487) and
// update at four elements; stage 1 also forms the factors
// (evolution.f90:604-607).  kt: the elements in the tables (i less the
// member's offset).
template <int STAGE>
__device__ __forceinline__ void fs_rk_qd(const FsEndArgs &a, const Scalars &sm,
                                         const long long (&i)[4], const long long (&kt)[4],
                                         double (&x)[4]) {
  if (a.heating || a.friction) {
    double p[4], q[4];
#pragma unroll
    for (int e = 0; e < 4; e++) {
      p[e] = a.pp[i[e]];
      q[e] = a.qq[i[e]];
    }
#pragma unroll
    for (int e = 0; e < 4; e++) {
      if (a.heating && !a.friction)
        x[e] = x[e] + a.therm * (p[e] - 0.0);
      else if (a.heating)
        x[e] = x[e] + a.therm * (p[e] - 0.0) - a.rekman * (q[e] + a.kdsq * p[e]);
      else
        x[e] = x[e] - a.rekman * (q[e] + a.kdsq * p[e]);
    }
  }
  double ep[4], em[4], d0[4], df[4];
#pragma unroll
  for (int e = 0; e < 4; e++) {
    if (STAGE == 1) {
      ep[e] = a.qdiss[kt[e]];
      d0[e] = a.qd[i[e]];
    } else {
      ep[e] = a.epq[i[e]];
      em[e] = a.emq[i[e]];
      if (STAGE != 4) d0[e] = a.qdi[i[e]];
      df[e] = a.qdf[i[e]];
    }
  }
  const double dt = sm.dt, dt2 = sm.dt2, dt3 = sm.dt3, dt6 = sm.dt6;
  const double dfac = dt2 * sm.zzrms;
#pragma unroll
  for (int e = 0; e < 4; e++) {
    if (STAGE == 1) {
      const double ex = exp(dfac * ep[e]), inv = 1.0 / ex;
      a.epq[i[e]] = ex;
      a.emq[i[e]] = inv;
      a.qdi[i[e]] = d0[e];
      a.qd[i[e]] = inv * (d0[e] + dt2 * x[e]);
      a.qdf[i[e]] = d0[e] + dt6 * x[e];
    } else if (STAGE == 2) {
      const double y = ep[e] * x[e];
      a.qd[i[e]] = em[e] * (d0[e] + dt2 * y);
      a.qdf[i[e]] = df[e] + dt3 * y;
    } else if (STAGE == 3) {
      const double y = ep[e] * x[e], m2 = em[e] * em[e];
      a.emq[i[e]] = m2;
      a.qd[i[e]] = m2 * (d0[e] + dt * y);
      a.qdf[i[e]] = df[e] + dt3 * y;
    } else {
      const double y = ep[e] * ep[e] * x[e];
      a.qd[i[e]] = em[e] * (df[e] + dt6 * y);
    }
  }
}
// The node update of a stage (evolution.f90:212-311), and (COUNT) the next
// stage's con2grid count of the segments between the moved nodes, which is
// otherwise a launch of its own.  A warp then moves 32 nodes and owns the first
// 31 (the 32nd is the next warp's first again), so that a segment's far end,
// almost always the next node, comes from the next lane; the last segment of a
// contour moves its far end a second time.  Worth it while a launch costs its
// latency (64^2, 10k nodes: a step 232 to 217 us); with the nodes in a launch of
// their own it is not (1.4M nodes: 36 + 42 us apart, 76 together, at 46 and 70
// registers).
template <int STAGE>
__device__ __forceinline__ double2 moved(const NodeMoveArgs &a, const Scalars *__restrict__ sc,
                                         const Consts &c, int i, int m, double2 &u) {
  const Scalars &sm = sc[m];
  const long long nn = (long long)c.nx * c.ny;
  const double x = a.x[i], y = a.y[i];
  velint1(x, y, a.uu + m * nn, a.vv + m * nn, c, u.x, u.y);
  if (a.du) {
    u.x = u.x + a.du[i];
    u.y = u.y + a.dv[i];
  }
  const double h = STAGE == 3 ? sm.dt : (STAGE == 4 ? sm.dt6 : sm.dt2);
  const double bx = STAGE == 1 ? x : (STAGE == 4 ? a.xf[i] : a.x0[i]);
  const double by = STAGE == 1 ? y : (STAGE == 4 ? a.yf[i] : a.y0[i]);
  return make_double2(wrapp(bx + h * u.x, c.ellx, c.hlxi, c.oms),
                      wrapp(by + h * u.y, c.elly, c.hlyi, c.oms));
}
template <int STAGE, bool COUNT>
__device__ __forceinline__ void move_nodes(int bid, int nbk, const NodeMoveArgs &a,
                                           const Scalars *__restrict__ sc, const Consts &c) {
  constexpr int OWN = COUNT ? 31 : 32;
  const unsigned FULL = 0xffffffffu;
  const int npt = sc->nptq, lane = threadIdx.x & 31, nw = nbk * (blockDim.x >> 5);
  if (COUNT && a.JW && bid == 0)  // the coarsening that follows accumulates here
    for (int m = threadIdx.x; m < a.mb.M; m += blockDim.x) a.csum[(long long)m * a.mb.cs] = 0;
  for (long long base = (long long)(bid * (blockDim.x >> 5) + (threadIdx.x >> 5)) * OWN; base < npt;
       base += (long long)nw * OWN) {
    const int i = (int)base + lane;
    const bool own = lane < OWN && i < npt;
    int ia = -1, m = 0;
    double2 u, p = make_double2(0.0, 0.0);
    if (i < npt) {
      if (COUNT && a.JW && own) ia = a.nextq[i];
      m = member_of(a.mb.mnode, a.mb.M, i);
      p = moved<STAGE>(a, sc, c, i, m, u);
    }
    if (own) {
      a.xn[i] = p.x;
      a.yn[i] = p.y;
      if (STAGE < 4) {
        const double h = STAGE == 1 ? sc[m].dt6 : sc[m].dt3;
        const double fx = STAGE == 1 ? a.x0[i] : a.xf[i], fy = STAGE == 1 ? a.y0[i] : a.yf[i];
        a.xf[i] = wrapp(fx + h * u.x, c.ellx, c.hlxi, c.oms);
        a.yf[i] = wrapp(fy + h * u.y, c.elly, c.hlyi, c.oms);
      }
    }
    if (COUNT && a.JW) {
      double2 q = make_double2(__shfl_down_sync(FULL, p.x, 1), __shfl_down_sync(FULL, p.y, 1));
      if (own) {
        if (ia < 0 || ia >= npt) {
          atomicExch(a.err, CASL_EINVAL);
        } else {
          if (ia != i + 1) q = moved<STAGE>(a, sc, c, ia, m, u);
          c2g_segment<true>(p.x, p.y, q.x, q.y, nullptr, a.JW + (long long)m * a.mb.jws,
                            a.ljx + (long long)m * a.mb.ljs, c, a.err);
        }
      }
    }
  }
}

template <int LOGN, int STAGE>
__global__ void __launch_bounds__(FsEnd<LOGN>::NT, 1024 / FsEnd<LOGN>::NT)
    k_fs_end(FsEndArgs a, NodeMoveArgs nd, Scalars *__restrict__ sc, Consts c, int nbn,
             const double2 *__restrict__ tw) {
  CASL_PDL_ENTRY();
  using Sh = FsEnd<LOGN>;
  constexpr int N = Sh::N, TPV = Sh::TPV, P = Sh::P, SL = fs_slot<LOGN>();
  constexpr long long nn = (long long)N * N;
  // the half-step time advance that opens stages 2 and 4 (nothing reads t
  // in between)
  if ((STAGE == 1 || STAGE == 3) && blockIdx.x == 0)
    for (int m = threadIdx.x; m < nd.mb.M; m += blockDim.x) sc[m].t = sc[m].t + sc[m].dt2;
  const int nrow = gridDim.x - nbn;
  if ((int)blockIdx.x >= nrow) {
    move_nodes<STAGE, (STAGE < 4)>(blockIdx.x - nrow, nbn, nd, sc, c);
    return;
  }
  extern __shared__ double2 smem[];
  const int mem = blockIdx.x / Sh::ROWB, rb = blockIdx.x - mem * Sh::ROWB;
  const int grp = threadIdx.x / TPV, t = threadIdx.x - grp * TPV;
  const int f = grp & 1, r0 = 2 * (rb * P + (grp >> 1));
  const long long o = mem * nn + (long long)r0 * N;
  double2 *S = smem + grp * SL;
  auto at = [&](int i) -> double2 & { return S[cpad(i)]; };
  auto sync = [&] { group_sync<TPV>(grp); };
  if (t == 0) {
    constexpr uint32_t by = 2 * N * 8;
    if (f == 0) {
      if (STAGE == 1) {
        l2_prefetch(a.qd + o, by);
        l2_prefetch(a.qdiss + (long long)r0 * N, by);
      } else {
        if (STAGE != 4) l2_prefetch(a.qdi + o, by);
        l2_prefetch(a.qdf + o, by);
        l2_prefetch(a.emq + o, by);
        l2_prefetch(a.epq + o, by);
      }
    } else if (STAGE == 1) {
      l2_prefetch(a.qs + o, by);
    } else {
      if (STAGE != 4) l2_prefetch(a.qsi + o, by);
      l2_prefetch(a.qsf + o, by);
    }
  }
  const double *T0 = a.tp + (mem * 2 + f) * nn + (long long)r0 * N;
  double2 x[8];
#pragma unroll
  for (int m = 0; m < 8; m++) {
    const int j = t + m * TPV;
    x[m] = make_double2(T0[j], T0[N + j]);
  }
  cfft<LOGN, true>(x, t, tw, at, sync);
#pragma unroll
  for (int m = 0; m < 8; m++) at(t + m * TPV) = x[m];
  sync();
  const double s = 1.0 / sqrt((double)N);
  const Scalars &sm = sc[mem];
  const long long kt = (long long)r0 * N;
#pragma unroll
  for (int m = 0; m < 4; m++) {
    const int k = t + m * TPV;
    double2 lo, hi;
    if (k == 0) {
      const double2 z0 = at(0), zh = at(N / 2);
      lo = make_double2(z0.x * s, z0.y * s);
      hi = make_double2(zh.x * s, zh.y * s);
    } else {
      fs_untangle(at(k), at(N - k), s, lo, hi);
    }
    const int kh = k == 0 ? N / 2 : N - k;
    const long long i[4] = {o + k, o + N + k, o + kh, o + N + kh};
    double v[4] = {lo.x, lo.y, hi.x, hi.y};
    if (f) {
      fs_rk_qs<STAGE>(a, sm, i, v);
    } else {
      const long long q[4] = {kt + k, kt + N + k, kt + kh, kt + N + kh};
      fs_rk_qd<STAGE>(a, sm, i, q, v);
    }
  }
}

// The node update alone: 46 registers, so 1280 nodes in flight per SM where
// k_fs_end's blocks hold 1024 threads.  Up to 148 * 1024 nodes all fit at once
// beside the rows and one launch is cheaper (64^2, 10k nodes: 275 against
// 280 us a step); above, the gathers' latency decides (512^2, 0.94M nodes: 15 +
// 24 us apart against 45 us together; 1024^2, 1.4M nodes: 27 + 36 against 55).
#define FS_NODES_TOGETHER (148 * 1024)
template <int STAGE>
__global__ void __launch_bounds__(256)
    k_nodes_rk(NodeMoveArgs nd, const Scalars *__restrict__ sc, Consts c) {
  CASL_PDL_ENTRY();
  move_nodes<STAGE, false>(blockIdx.x, gridDim.x, nd, sc, c);
}

}  // namespace casl

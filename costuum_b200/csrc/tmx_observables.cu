// Observables of (orientation-averaged) T-matrices on device (sm_100a, FP64).
//
//   k_cg            Clebsch-Gordan rows <n1 m n2 -m | N 0>, m >= 0
//                   (SpecialFunctions::get_clebsch_gordan_coefficients,
//                   SpecialFunctions.hpp:1131-1244)
//   k_orient        AlignmentAverageTask::execute (AlignmentAverageTask.hpp:
//                   115-215), restructured: the m1 sum does not depend on m,
//                   so it is formed once per (n1, n2, N) and reused for every
//                   m (O(N^4) instead of O(N^5))
//   k_amp           the per-m sums of the forward-scattering amplitude S of
//                   ExtinctionCoefficientTask.hpp:517-619 (and its copies in
//                   AbsorptionCoefficientTask.hpp:612-715 and
//                   ScatteringMatrixTask.hpp:588-691): T times the vectors of
//                   a set of incoming angles on the FP64 tensor pipe, then
//                   the product with each pair's outgoing vector
//   k_azimuth       S of every pair and azimuth from those sums, O(nmax) each
//   k_q_epilogue    Q_ext/Q_extpol/Q_extcpol and Q_abs/Q_abspol (with the
//                   optional scattering subtraction of
//                   AbsorptionCoefficientTask.hpp:742-773)
//   k_z_epilogue    4x4 scattering matrix (ScatteringMatrixTask.hpp:719-748)
//   k_shape_avg     ShapeAveragingTask (ShapeAveragingTask.hpp:127-166)
//
// Compiled with --fmad=false, like the table kernels, so the recurrences
// round as the reference's build does.
#include <algorithm>

#include "tmx_common.cuh"
#include "tmx_kernels.h"

// ---------------------------------------------------------- CG table -----

// offset table: cg_off[(n1 - 1) * nmax + (n2 - 1)] -> start of the pair's
// rows; row N (|n1-n2| <= N <= n1+n2) holds min(n1,n2) + 1 values, m = 0..min
__device__ static void cg_row(int nmax, int pair, int Ni,
                              const int64_t *__restrict__ cg_off,
                              double *__restrict__ cg, double *rowA,
                              double *rowB) {
  const int n1 = pair / nmax + 1;
  const int n2 = pair % nmax + 1;
  const int M = min(n1, n2);
  const int Nlo = abs(n1 - n2);
  const int N = Nlo + Ni;
  if (N > n1 + n2) {
    return;
  }
  const int nsize = 2 * n1 + 1;
  for (int i = 0; i < nsize; ++i) {
    rowA[i] = 0.;
    rowB[i] = 0.;
  }
  // upper row M = N
  double *top = rowA;
  top[n1 + n1] = 1.;
  double norm = 1.;
  const int lo = max(-n1, N - n2 - 1);
  for (int m1t = n1 - 1; m1t >= lo; --m1t) {
    const double cp2 = sqrt((n2 - N + m1t + 1.) * (n2 + N - m1t));
    const double cp1 = sqrt((n1 - m1t) * (n1 + m1t + 1.));
    const double cnext = -cp2 * top[m1t + 1 + n1] / cp1;
    top[m1t + n1] = cnext;
    norm += cnext * cnext;
  }
  const double inv_norm = 1. / sqrt(norm);
  for (int m1t = n1; m1t >= lo; --m1t) {
    top[m1t + n1] *= inv_norm;
  }
  double *prev = rowA, *cur = rowB;
  for (int Mt = N - 1; Mt >= 0; --Mt) {
    const double cmin_inv = 1. / sqrt((N + Mt + 1.) * (N - Mt));
    const int a = max(-n1, Mt - n2);
    const int b = min(n1, Mt + n2);
    for (int m1t = a; m1t <= b; ++m1t) {
      const int m2t = Mt - m1t;
      double t1 = 0.;
      if (m1t + 1 <= n1) {
        t1 = sqrt((n1 + m1t + 1.) * (n1 - m1t)) * prev[m1t + 1 + n1];
      }
      double t2 = 0.;
      if (m2t + 1 <= n2) {
        t2 = sqrt((n2 + m2t + 1.) * (n2 - m2t)) * prev[m1t + n1];
      }
      cur[m1t + n1] = cmin_inv * (t1 + t2);
    }
    double *t = prev;
    prev = cur;
    cur = t;
  }
  // prev holds row M = 0; keep m = 0..M
  double *o = cg + cg_off[pair] + (int64_t)(N - Nlo) * (M + 1);
  for (int m = 0; m <= M; ++m) {
    o[m] = prev[m + n1];
  }
}

__global__ void k_cg(int nmax, const int64_t *__restrict__ cg_off,
                     double *__restrict__ cg, double *__restrict__ work) {
  const int npairs = nmax * nmax;
  const int rows = 2 * nmax + 1; // at most 2 nmax + 1 values of N per pair
  const int slot = blockIdx.x * blockDim.x + threadIdx.x;
  const int wlen = 2 * nmax + 1;
  // two rolling rows of the ladder recursion in this thread's work slot
  double *rowA = work + (int64_t)slot * 2 * wlen;
  double *rowB = rowA + wlen;
  for (int64_t u = slot; u < (int64_t)npairs * rows;
       u += (int64_t)gridDim.x * blockDim.x) {
    cg_row(nmax, (int)(u / rows), (int)(u % rows), cg_off, cg, rowA, rowB);
  }
}

// ------------------------------------------------- orientation average ---

__device__ __forceinline__ int64_t tblock(int N, int m) {
  if (m == 0) {
    return 0;
  }
  const int64_t a = N, b = N + 1 - m;
  return 4 * (a * a + a * (a + 1) * (2 * a + 1) / 6 - b * (b + 1) * (2 * b + 1) / 6);
}

// element (i1, n1; i2, n2) of block m of a T-matrix of order N
__device__ __forceinline__ int64_t telem(int N, int m, int i1, int n1, int i2,
                                         int n2) {
  const int nb = (m == 0) ? N : N + 1 - m;
  const int nmin = (m == 0) ? 1 : m;
  return tblock(N, m) + (int64_t)(i1 * nb + n1 - nmin) * (2 * nb) + i2 * nb +
         n2 - nmin;
}

// matrix k of a set (selects, so that the pointers stay in constant memory)
__device__ __forceinline__ const cplx *mat_src(const TmxMatSet &s, int k) {
  return k == 0 ? s.src[0] : k == 1 ? s.src[1] : k == 2 ? s.src[2] : s.src[3];
}
__device__ __forceinline__ cplx *mat_dst(const TmxMatSet &s, int k) {
  return k == 0 ? s.dst[0] : k == 1 ? s.dst[1] : k == 2 ? s.dst[2] : s.dst[3];
}

// acc += t * a (complex times real), fused; this file is compiled without
// automatic contraction, so the contractions are spelled out
__device__ __forceinline__ void cfma(cplx &acc, cplx t, double a) {
  acc.x = __fma_rn(t.x, a, acc.x);
  acc.y = __fma_rn(t.y, a, acc.y);
}

// sqrt((2n + 1) / ((n + 1) n)), the factor of a_{n n'} for one order
__device__ __forceinline__ double a_fac(int n) {
  return sqrt((2. * n + 1.) / ((n + 1.) * n));
}

// element (i1, n1; i2, n2) of block m of an averaged T-matrix of order N in
// the compact class layout the amplitude kernel reads: the entries of the
// parity classes (i + n) % 2 of block m (m = 0: of each (i, n % 2)) one after
// the other as dense row-major matrices, members by i, then n. Half the size
// of the block; -1 for the entries between classes, which are zero.
__device__ __forceinline__ int64_t celem(int N, int m, int i1, int n1, int i2,
                                         int n2) {
  if (((i1 + n1 + i2 + n2) & 1) || (m == 0 && i1 != i2)) {
    return -1;
  }
  if (m == 0) {
    const int no = (N + 1) >> 1, ne = N >> 1;
    const int ld = (n1 & 1) ? no : ne;
    const int64_t off = (int64_t)i1 * (no * no + ne * ne) + ((n1 & 1) ? 0 : no * no);
    return off + (int64_t)((n1 - 1) >> 1) * ld + ((n2 - 1) >> 1);
  }
  const int cls = (i1 + n1) & 1;
  const int L = N + 1 - m;
  // first order of the members with i = 0 and i = 1, and their number
  const int f0 = m + ((m & 1) != cls), f1 = m + ((m & 1) == cls);
  const int r0 = (N >= f0) ? (N - f0) / 2 + 1 : 0;
  const int a = i1 ? r0 + ((n1 - f1) >> 1) : (n1 - f0) >> 1;
  const int b = i2 ? r0 + ((n2 - f1) >> 1) : (n2 - f0) >> 1;
  return tblock(N, m) / 2 + ((int64_t)cls * L + a) * L + b;
}

// c_{n' n} z for c_{n' n} = i^{n' - n - 1} a_{n' n} (NBasedResources::get_cnn,
// NBasedResources.hpp:115-137); n' is the incoming order (column), n the
// outgoing one (row)
__device__ __forceinline__ cplx c_fold(int nin, int nout, double a, cplx z) {
  const cplx s = cscale(z, a);
  switch ((((nin - nout - 1) % 4) + 4) % 4) {
  case 0:
    return s;
  case 1:
    return mkc(-s.y, s.x);
  case 2:
    return mkc(-s.x, -s.y);
  default:
    return mkc(s.y, -s.x);
  }
}

// D += A B for one m8n8k4 FP64 tensor-core tile: lane l holds A[l / 4][l % 4],
// B[l % 4][l / 4] and D[l / 4][2 (l % 4) + {0, 1}]
__device__ __forceinline__ void dmma(double &d0, double &d1, double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, "
      "{%0, %1};\n"
      : "+d"(d0), "+d"(d1)
      : "d"(a), "d"(b));
}

// AlignmentAverageTask::execute (AlignmentAverageTask.hpp:115-215) forms, for
// every m,
//   Ta_m = sum_N' p_N' (-1)^m CG(n1 m n2 -m|N'0) sum_m1 f(m1) (-1)^m1
//          CG(n1 m1 n2 -m1|N'0) T_m1,
// with f = 1 for m1 = 0 and 2 otherwise; the m1 sum does not depend on m, so
// pass 1 forms it once per N' and pass 2 contracts over N': O(n^2) per pair
// instead of O(n^3). T couples (0,0) and (1,1) for even n1 + n2 and (0,1) and
// (1,0) for odd ones, and only the N' of that parity contribute, so of the two
// sub-block pairs and the 2 M + 1 rows of the Clebsch-Gordan table one half is
// left (M = min(n1, n2)).
//
// One warp per (pair, chunk of 2 NT grains): both passes are products of the
// pair's Clebsch-Gordan rows with 8 NT real columns (grain, sub-block, re/im)
// on the FP64 tensor pipe; t and S = p_N' CG t go through shared memory, whose
// rows are 4 doubles off a multiple of 16 (the fragments' 4 x 4 doubles hit
// distinct banks). A chunk shares each row it reads, so the table is read once
// per 2 NT grains. Grains without an orientation distribution (coef_set < 0)
// are copied. With fold the output carries the factor c_{n2 n1} of the
// amplitude sums, so that the amplitude kernel contracts with real vectors.
// Measured (B200), one warp per (pair, grain) with FMA dot products over all
// rows and sub-blocks -> this kernel: 96 grains of orders 16..50 0.59 -> 0.23
// ms; 1920 grains of orders 10..99 6.7 -> 2.9 ms; 1024 grains and their three
// tangents 1.44 -> 0.54 ms. Bound by the scattered 16-byte T reads (half of
// each sector) and, above order 63, by the table reads of few grains.
template <int NT>
__global__ void __launch_bounds__(128)
k_orient(const TmxObsGrain *__restrict__ og, const int32_t *__restrict__ order,
         const TmxOrientRange *__restrict__ rng, int nrng, int64_t nitems, int ncap,
         TmxMatSet mats, const double *__restrict__ coeffs, int ncoef,
         const int64_t *__restrict__ cg_off, const double *__restrict__ cg,
         int cg_nmax, int fold) {
  constexpr int G = 2 * NT;       // grains per chunk
  constexpr int LD = 8 * NT + 4;  // row of t and S
  constexpr int CB = 8;           // table entries in flight per lane
  extern __shared__ double osm[];
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  const int q = lane & 3;
  const int rr = lane >> 2;
  const int64_t w = (int64_t)blockIdx.x * 4 + warp;
  if (w >= nitems) {
    return;
  }
  const int rows = (ncap + 7) & ~7;
  double *t = osm + (int64_t)warp * 2 * rows * LD; // [m][LD]
  double *S = t + rows * LD;                       // [N'][LD]
  int lo = 0, hi = nrng - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (rng[mid].base <= w) {
      lo = mid;
    } else {
      hi = mid - 1;
    }
  }
  const TmxOrientRange R = rng[lo];
  const int nch = (R.ng + G - 1) / G;
  const int pr = (int)((w - R.base) / nch);
  const int g0 = (int)((w - R.base) % nch) * G;
  const int n1 = (pr < R.n) ? R.n : pr - R.n + 1;
  const int n2 = (pr < R.n) ? pr + 1 : R.n;
  const int M = min(n1, n2);
  const int par = (n1 + n2) & 1;
  const cplx *src = mat_src(mats, blockIdx.y);
  cplx *dst = mat_dst(mats, blockIdx.y);
  // t[m][4 grain + 2 block + re/im]: block 0 is (0, par), block 1 (1, 1 - par)
  bool avg_any = false;
  {
    const int e = lane % (2 * G);
    const int blk = e & 1;
    const bool have = g0 + (e >> 1) < R.ng;
    const TmxObsGrain gr = og[order[have ? g0 + (e >> 1) : 0]];
    const bool avg = have && gr.coef_set >= 0;
    avg_any = __any_sync(0xffffffffu, avg);
    for (int m = lane / (2 * G); m < ((M + 4) & ~3); m += 32 / (2 * G)) {
      cplx v = mkc(0., 0.);
      if (have && m <= M) {
        v = src[gr.t_off + telem(gr.nmax, m, blk, n1, blk ^ par, n2)];
        // f(m) (-1)^m is a power of two with a sign: the product is exact
        const double f = avg ? ((m == 0) ? 1. : 2.) * ((m & 1) ? -1. : 1.) : 1.;
        v = cscale(v, f);
      }
      *reinterpret_cast<cplx *>(t + m * LD + 2 * e) = v;
    }
  }
  __syncwarp();
  // (no table where nothing is averaged)
  const double *C = avg_any ? cg + cg_off[(n1 - 1) * cg_nmax + (n2 - 1)] : nullptr;
  const int nrow = M + 1 - par; // N' of the pair's parity: j = 2 jr + par
  // the grains of this lane's output columns
  int gN[NT], gset[NT];
  int64_t goff[NT];
#pragma unroll
  for (int j = 0; j < NT; ++j) {
    const int g = g0 + 2 * j + (q >> 1);
    gN[j] = 0;
    gset[j] = -1;
    goff[j] = 0;
    if (g < R.ng) {
      const TmxObsGrain gr = og[order[g]];
      gN[j] = gr.nmax;
      gset[j] = gr.coef_set;
      goff[j] = gr.t_off;
    }
  }
  if (avg_any) {
    // pass 1: S(N') = p_N' sum_m1 CG t
    const int Nlo = abs(n1 - n2);
    for (int r0 = 0; r0 < nrow; r0 += 8) {
      const int jr = r0 + rr;
      const double *Cr = C + (int64_t)(2 * jr + par) * (M + 1);
      double acc[NT][2];
#pragma unroll
      for (int j = 0; j < NT; ++j) {
        acc[j][0] = acc[j][1] = 0.;
      }
      for (int k0 = 0; k0 <= M; k0 += 4 * CB) {
        double a[CB];
#pragma unroll
        for (int b = 0; b < CB; ++b) {
          const int m = k0 + 4 * b + q;
          a[b] = (jr < nrow && m <= M) ? Cr[m] : 0.;
        }
#pragma unroll
        for (int b = 0; b < CB; ++b) {
          if (k0 + 4 * b <= M) {
            const double *tb = t + (k0 + 4 * b + q) * LD + rr;
#pragma unroll
            for (int j = 0; j < NT; ++j) {
              dmma(acc[j][0], acc[j][1], a[b], tb[8 * j]);
            }
          }
        }
      }
#pragma unroll
      for (int j = 0; j < NT; ++j) {
        const double p = (jr < nrow && gset[j] >= 0)
                             ? coeffs[(int64_t)gset[j] * ncoef + Nlo + 2 * jr + par]
                             : 0.;
        *reinterpret_cast<double2 *>(S + jr * LD + 8 * j + 2 * q) =
            make_double2(acc[j][0] * p, acc[j][1] * p);
      }
    }
    __syncwarp();
  }
  // pass 2: Ta_m = (-1)^m sum_N' CG S
  const double afold = fold ? a_fac(n1) * a_fac(n2) : 1.;
  const int nfold = fold ? n1 : n2 - 1; // (c = 1: i^0 times 1)
  const int i1 = q & 1, i2 = i1 ^ par;
  for (int m0 = 0; m0 <= M; m0 += 8) {
    const int m = m0 + rr;
    double acc[NT][2];
#pragma unroll
    for (int j = 0; j < NT; ++j) {
      acc[j][0] = acc[j][1] = 0.;
    }
    for (int k0 = 0; avg_any && k0 < nrow; k0 += 4 * CB) {
      double a[CB];
#pragma unroll
      for (int b = 0; b < CB; ++b) {
        const int jr = k0 + 4 * b + q;
        a[b] = (m <= M && jr < nrow) ? C[(int64_t)(2 * jr + par) * (M + 1) + m] : 0.;
      }
#pragma unroll
      for (int b = 0; b < CB; ++b) {
        if (k0 + 4 * b < nrow) {
          const double *sb = S + (k0 + 4 * b + q) * LD + rr;
#pragma unroll
          for (int j = 0; j < NT; ++j) {
            dmma(acc[j][0], acc[j][1], a[b], sb[8 * j]);
          }
        }
      }
    }
    if (m > M || (m == 0 && i1 != i2)) {
      continue;
    }
    const double ms = (m & 1) ? -1. : 1.;
#pragma unroll
    for (int j = 0; j < NT; ++j) {
      if (gN[j] > 0) {
        const cplx v = (gset[j] >= 0)
                           ? mkc(ms * acc[j][0], ms * acc[j][1])
                           : *reinterpret_cast<const cplx *>(t + m * LD + 8 * j + 2 * q);
        const int64_t o = fold ? goff[j] / 2 + celem(gN[j], m, i1, n1, i2, n2)
                               : goff[j] + telem(gN[j], m, i1, n1, i2, n2);
        dst[o] = c_fold(n2, nfold, afold, v);
      }
    }
  }
}

// -------------------------------------------------- forward amplitude ----

// pi_n = m d^n_{0m}(x) / sin x and tau_n = d/dx d^n_{0m}(x) for one m and
// n = nmin..nmax, written to pi[(n - nmin) * stride], tau[...]
// (SpecialFunctions::wigner_dn_0m_sinx, SpecialFunctions.hpp:397-495)
__device__ static void wigner_col(double cosx, double sinx, double sinx_inv,
                                  int nmax, int m, double *pi, double *tau,
                                  int stride) {
  const int nmin = (m > 1) ? m : 1;
  if (fabs(1. - fabs(cosx)) <= 1.e-10) {
    if (m == 1) {
      int sign = 1;
      for (int n = 1; n < nmax + 1; ++n) {
        double dn = 0.5 * sqrt(n * (n + 1.));
        if (cosx < 0.) {
          dn *= sign;
        }
        pi[(n - nmin) * stride] = m * dn;
        if (cosx < 0.) {
          dn = -dn;
        }
        tau[(n - nmin) * stride] = dn;
        sign = -sign;
      }
    } else {
      for (int n = nmin; n <= nmax; ++n) {
        pi[(n - nmin) * stride] = 0.;
        tau[(n - nmin) * stride] = 0.;
      }
    }
    return;
  }
  if (m == 0) {
    double d1 = 1.;
    double d2 = cosx;
#pragma unroll 4
    for (int n = 0; n < nmax; ++n) {
      const double np1 = n + 1.;
      const double np2 = n + 2.;
      const double np12p1 = 2. * np1 + 1.;
      const double r2 = 1. / np2;
      const double dnp1 = __fma_rn(np12p1 * cosx * r2, d2, -(np1 * r2 * d1));
      const double ddn = (sinx_inv * np1 * np2 / np12p1) * (dnp1 - d1);
      pi[n * stride] = 0.;
      tau[n * stride] = ddn;
      d1 = d2;
      d2 = dnp1;
    }
    return;
  }
  // the square roots and quotients of a step do not depend on the step before
  // it: only one fused multiply-add per order is serial
  const double m2 = (double)(m * m);
  double d1 = 0.;
  double d2 = 1.;
#pragma unroll 4
  for (int i = 0; i < m; ++i) {
    const double i2 = 2. * (i + 1.);
    d2 *= sqrt((i2 - 1.) / i2) * sinx;
  }
  double s12 = 0.; // sqrt(n^2 - m^2) at n = m
#pragma unroll 4
  for (int n = m - 1; n < nmax; ++n) {
    const double np1 = n + 1.;
    const double np2 = n + 2.;
    const double np12p1 = 2. * np1 + 1.;
    const double s22 = sqrt(np2 * np2 - m2);
    const double r22 = 1. / s22;
    const double dnp1 = __fma_rn(np12p1 * cosx * r22, d2, -(s12 * r22 * d1));
    const double ddn =
        (sinx_inv / np12p1) * (np1 * s22 * dnp1 - np2 * s12 * d1);
    pi[(n + 1 - nmin) * stride] = m * (d2 * sinx_inv);
    tau[(n + 1 - nmin) * stride] = ddn;
    d1 = d2;
    d2 = dnp1;
    s12 = s22;
  }
}

// pi and tau columns of every (angle, m <= nmax) of an amplitude plan, once
// for all grains and jobs that share an angle: column (a, m) holds orders n = max(m, 1) .. nmax at ((a (nmax + 1) + m)
// nmax). (The values of orders <= N do not depend on how far the
// recurrence runs, so a grain of order N reads the first entries.)
__global__ void k_wigner_cols(const TmxAngle *__restrict__ angles, int nangles,
                              int nmax, double *pi, double *tau) {
  const int64_t u = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (u >= (int64_t)nangles * (nmax + 1)) {
    return;
  }
  const int a = (int)(u / (nmax + 1));
  const int m = (int)(u - (int64_t)a * (nmax + 1));
  const TmxAngle A = angles[a];
  wigner_col(A.c, A.s, A.si, nmax, m, pi + u * nmax, tau + u * nmax, 1);
}

// parity class c of block m of order N: members (i = 0, n = f0 + 2 j), j <
// r0, then (i = 1, n = f1 + 2 j), nb in all (celem's order), and its offset
struct AmpClass {
  int nb, r0, f0, f1;
  int64_t off;
};
__device__ __forceinline__ AmpClass amp_class(int N, int m, int c) {
  AmpClass A;
  if (m == 0) {
    const int no = (N + 1) >> 1, ne = N >> 1;
    A.f0 = A.f1 = 1 + (c & 1);
    A.nb = (c & 1) ? ne : no;
    A.r0 = (c >> 1) ? 0 : A.nb;
    A.off = (int64_t)(c >> 1) * (no * no + ne * ne) + ((c & 1) ? no * no : 0);
    return A;
  }
  A.nb = N + 1 - m;
  A.f0 = m + ((m & 1) != c);
  A.f1 = m + ((m & 1) == c);
  A.r0 = (N >= A.f0) ? (N - A.f0) / 2 + 1 : 0;
  A.off = tblock(N, m) / 2 + (int64_t)c * A.nb * A.nb;
  return A;
}

// One CTA per (group, block m): with u = (pi_n, tau_n) at the outgoing angle
// and v at the incoming one (n the row order, n' the column order of block m),
//   X0 = u^T Tc v,  X1 = u^T Tc v',  X2 = u'^T Tc v,  X3 = u'^T Tc v'
// where Tc is block m with the c_{n' n} factors folded in and u', v' swap
// the pi and tau halves: the four (n, n') sums of
// ExtinctionCoefficientTask.hpp:517-619.
// Phase 1 forms y = Tc v, y' = Tc v' of every incoming angle: per parity class
// an (nb x nb) complex by (nb x 2 nin) real product, 8-row tiles over the
// warps, columns (angle, v or v') on the FP64 tensor pipe, T entries straight
// from memory (each is used once per CTA), eight K steps in flight. Phase 2
// multiplies with the outgoing vectors pair by pair, 2^k lanes per pair.
// Splitting over m (rather than one CTA looping over a grain's blocks) fills
// the chip from a few grains on, and an incoming angle's product is formed
// once however many outgoing angles it goes with. Only the entries of the
// parity classes are read (half of a block, the rest is zero).
// Measured (B200): 96 grains of orders 16..50, 16 angles: 2.11 ms with one CTA
// of FMA dot products per grain -> 0.093 ms; a 1920-grain table, orders 10..99,
// 32 angles: 29.0 -> 0.84 ms; the three tangents of 1024 grains, 32 angles:
// 1.92 -> 0.72 ms. Bound by the latency of the T reads and of phase 2's
// shared-memory reads at small L, well below the FP64 and HBM rates.
template <int NT, int NTH>
__global__ void __launch_bounds__(NTH, (NTH == 128) ? 4 : 2)
k_amp(const TmxAmpGroup *__restrict__ groups, const int32_t *__restrict__ ins,
      const TmxAmpPair *__restrict__ pairs, const TmxAmpRange *__restrict__ rng,
      int nrng, const TmxObsGrain *__restrict__ og, TmxMatSet mats,
      const double *__restrict__ wpi, const double *__restrict__ wtau, int wnmax,
      cplx *__restrict__ X, int64_t xstride, int lcap) {
  constexpr int NA = 4 * NT;              // angle slots
  constexpr int VS = (NA > 8) ? 18 : 10;  // row stride: k steps of 2 orders hit
                                          // distinct bank groups
  extern __shared__ cplx ash[];
  cplx *Y = ash;                          // [2 L][NA][2]: row (i, n), (y, y')
  double *V = reinterpret_cast<double *>(Y + (int64_t)2 * lcap * NA * 2); // [2][L][VS]
  const int tid = threadIdx.x;
  const int lane = tid & 31;
  const int warp = tid >> 5;
  int lo = 0, hi = nrng - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (rng[mid].base <= (int64_t)blockIdx.x) {
      lo = mid;
    } else {
      hi = mid - 1;
    }
  }
  const TmxAmpRange R = rng[lo];
  const int m = R.m;
  const TmxAmpGroup grp = groups[R.first + (int)(blockIdx.x - R.base)];
  const TmxObsGrain G = og[grp.grain];
  const int N = G.nmax;
  const int nmin = (m > 1) ? m : 1;
  const int L = N + 1 - nmin;
  const cplx *T = mat_src(mats, blockIdx.y) + G.t_off / 2;
  // incoming vectors: V[0] = pi, V[1] = tau
  for (int u = tid; u < NA * L; u += NTH) {
    const int a = u / L;
    const int k = u - a * L;
    double p = 0., t = 0.;
    if (a < grp.nin) {
      const int64_t off = ((int64_t)ins[grp.in0 + a] * (wnmax + 1) + m) * wnmax + k;
      p = wpi[off];
      t = wtau[off];
    }
    V[k * VS + a] = p;
    V[(L + k) * VS + a] = t;
  }
  __syncthreads();
  {
    const int rr = lane >> 2;
    const int kq = lane & 3;
    const int ncls = (m == 0) ? 4 : 2;
    int tile0 = 0; // tiles of the classes before this one
    for (int c = 0; c < ncls; ++c) {
      const AmpClass C = amp_class(N, m, c);
      const int nrt = (C.nb + 7) >> 3;
      const cplx *Tc = T + C.off;
      // this warp's row tiles of the class
      for (int rt = (warp - tile0 % (NTH / 32) + NTH / 32) % (NTH / 32); rt < nrt;
           rt += NTH / 32) {
        double acc[NT][4];
#pragma unroll
        for (int j = 0; j < NT; ++j) {
          acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.;
        }
        const int row = rt * 8 + rr;
        const cplx *Tr = Tc + (int64_t)row * C.nb;
        for (int k0 = 0; k0 < C.nb; k0 += 32) {
          cplx t[8];
#pragma unroll
          for (int s = 0; s < 8; ++s) {
            const int col = k0 + 4 * s + kq;
            t[s] = (row < C.nb && col < C.nb) ? Tr[col] : mkc(0., 0.);
          }
#pragma unroll
          for (int s = 0; s < 8; ++s) {
            if (k0 + 4 * s < C.nb) {
              const int col = min(k0 + 4 * s + kq, C.nb - 1);
              const int i = (col < C.r0) ? 0 : 1;
              const int n = i ? C.f1 + 2 * (col - C.r0) : C.f0 + 2 * col;
              // column rr of the tile: angle rr / 2, v (0) or v' (1)
              const double *v = V + (((rr & 1) ^ i) * L + n - nmin) * VS + (rr >> 1);
#pragma unroll
              for (int j = 0; j < NT; ++j) {
                const double b = v[4 * j];
                dmma(acc[j][0], acc[j][1], t[s].x, b);
                dmma(acc[j][2], acc[j][3], t[s].y, b);
              }
            }
          }
        }
        if (row < C.nb) {
          const int i = (row < C.r0) ? 0 : 1;
          const int n = i ? C.f1 + 2 * (row - C.r0) : C.f0 + 2 * row;
          cplx *y = Y + ((int64_t)(i * L + n - nmin) * NA + kq) * 2;
#pragma unroll
          for (int j = 0; j < NT; ++j) {
            y[8 * j] = mkc(acc[j][0], acc[j][2]);
            y[8 * j + 1] = mkc(acc[j][1], acc[j][3]);
          }
        }
      }
      tile0 += nrt;
    }
  }
  __syncthreads();
  // lanes per pair: as many as keep every thread busy
  int ns = 1;
  while (ns < 32 && grp.npair * ns * 2 <= NTH) {
    ns *= 2;
  }
  const int sl = tid & (ns - 1);
  for (int p0 = 0; p0 < grp.npair; p0 += NTH / ns) {
    const int p = p0 + tid / ns;
    const bool act = p < grp.npair;
    const TmxAmpPair P = pairs[grp.pair0 + (act ? p : 0)];
    cplx x0 = mkc(0., 0.), x1 = x0, x2 = x0, x3 = x0;
    if (act) {
      const int64_t off = ((int64_t)P.angle_out * (wnmax + 1) + m) * wnmax;
      for (int k = sl; k < L; k += ns) {
        const double a = wpi[off + k], b = wtau[off + k];
        const cplx *y = Y + ((int64_t)k * NA + P.in) * 2;
        const cplx *z = y + (int64_t)L * NA * 2;
        const cplx y0 = y[0], y1 = y[1], z0 = z[0], z1 = z[1];
        cfma(x0, y0, a);
        cfma(x0, z0, b);
        cfma(x1, y1, a);
        cfma(x1, z1, b);
        cfma(x2, y0, b);
        cfma(x2, z0, a);
        cfma(x3, y1, b);
        cfma(x3, z1, a);
      }
    }
    for (int o = ns >> 1; o > 0; o >>= 1) {
      x0.x += __shfl_xor_sync(0xffffffffu, x0.x, o);
      x0.y += __shfl_xor_sync(0xffffffffu, x0.y, o);
      x1.x += __shfl_xor_sync(0xffffffffu, x1.x, o);
      x1.y += __shfl_xor_sync(0xffffffffu, x1.y, o);
      x2.x += __shfl_xor_sync(0xffffffffu, x2.x, o);
      x2.y += __shfl_xor_sync(0xffffffffu, x2.y, o);
      x3.x += __shfl_xor_sync(0xffffffffu, x3.x, o);
      x3.y += __shfl_xor_sync(0xffffffffu, x3.y, o);
    }
    if (act && sl == 0) {
      cplx *o = X + blockIdx.y * xstride + grp.x0 + ((int64_t)p * (N + 1) + m) * 4;
      o[0] = x0;
      o[1] = x1;
      o[2] = x2;
      o[3] = x3;
    }
  }
}

// S of every pair and azimuth of a group (blockIdx.x; blockIdx.y shares the
// azimuths of a group, blockIdx.z the matrices):
//   S = (1/k) sum_m (2 cos m phi, 2 sin m phi) X_m
// with e^{i m phi} built by repeated multiplication as in the reference.
__global__ void __launch_bounds__(128)
k_azimuth(const TmxAmpGroup *__restrict__ groups, const TmxAmpPair *__restrict__ pairs,
          const TmxObsGrain *__restrict__ og, TmxMatSet mats,
          const cplx *__restrict__ phis, const cplx *__restrict__ X, int64_t xstride) {
  const TmxAmpGroup grp = groups[blockIdx.x];
  const TmxObsGrain G = og[grp.grain];
  const int N = G.nmax;
  const double kinv = 1. / G.k;
  const TmxAmpPair *pr = pairs + grp.pair0;
  for (int item = blockIdx.y * blockDim.x + threadIdx.x; item < grp.nitem;
       item += gridDim.y * blockDim.x) {
    int lo = 0, hi = grp.npair - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (pr[mid].pref <= item) {
        lo = mid;
      } else {
        hi = mid - 1;
      }
    }
    const TmxAmpPair P = pr[lo];
    const int f = item - P.pref;
    const cplx e1 = phis[P.phi0 + f];
    const cplx *Xp = X + blockIdx.z * xstride + grp.x0 + (int64_t)lo * (N + 1) * 4;
    cplx s0 = Xp[0], s1 = mkc(0., 0.), s2 = s1, s3 = Xp[3];
    cplx e = cmul(mkc(1., 0.), e1);
#pragma unroll 4
    for (int m = 1; m <= N; ++m) {
      const double fcos = 2. * e.x;
      const double fsin = 2. * e.y;
      e = cmul(e, e1);
      const cplx *x = Xp + m * 4;
      s0 = cadd(s0, cscale(x[0], fcos));
      s1 = cadd(s1, cscale(x[1], fsin));
      s2 = csub(s2, cscale(x[2], fsin));
      s3 = cadd(s3, cscale(x[3], fcos));
    }
    cplx *o = mat_dst(mats, blockIdx.z) + (grp.out0 + P.out + f) * 4;
    o[0] = cscale(s0, kinv);
    o[1] = cscale(s1, kinv);
    o[2] = cscale(s2, kinv);
    o[3] = cscale(s3, kinv);
  }
}

// ----------------------------------------------------------- epilogues ---

__device__ __forceinline__ double zsum(const cplx *S, double s1, double s2,
                                       double s3) {
  // 0.5 (|S0|^2 + s1 |S1|^2 + s2 |S2|^2 + s3 |S3|^2)
  return 0.5 * (cnorm2(S[0]) + s1 * cnorm2(S[1]) + s2 * cnorm2(S[2]) +
                s3 * cnorm2(S[3]));
}

// One thread per (grain, theta), or with the scattering subtraction (ACC) one
// warp: extinction and absorption coefficients from the theta -> theta
// amplitude, minus the directional scattering integral when requested (the
// reference subtracts sum_{theta', phi'} w Z00 and Z10). The integral reads
// nacc^2 amplitudes of 64 bytes, so its lanes share them: 900 jobs of 400
// directions took 0.29 ms on one thread each, 0.014 ms on a warp.
template <bool ACC>
__global__ void k_q_epilogue(const TmxQJob *__restrict__ jobs, int njobs,
                             const TmxObsGrain *__restrict__ og,
                             const cplx *__restrict__ S,
                             const double *__restrict__ wts, int nacc,
                             double *__restrict__ qout, int qstride,
                             int do_abs, int do_ext) {
  const int lane = ACC ? threadIdx.x & 31 : 0;
  const int u = (blockIdx.x * blockDim.x + threadIdx.x) / (ACC ? 32 : 1);
  if (u >= njobs) {
    return;
  }
  const TmxQJob J = jobs[u];
  const TmxObsGrain G = og[J.grain];
  const cplx *s = S + J.s_main * 4;
  const double prefactor = 2. * M_PI / G.k;
  const double norm = M_PI * G.r_ev * G.r_ev;
  double *o = qout + (int64_t)J.out * qstride;
  int k = 0;
  if (do_abs) {
    double z0 = 0., z1 = 0.;
    if (ACC) {
#pragma unroll 2
      for (int i = lane; i < nacc * nacc; i += 32) {
        const cplx *st = S + (J.s_acc + i) * 4;
        const double w = wts[i / nacc] * wts[nacc + i % nacc];
        z0 += zsum(st, 1., 1., 1.) * w;
        z1 += zsum(st, 1., -1., -1.) * w;
      }
#pragma unroll
      for (int d = 16; d > 0; d >>= 1) {
        z0 += __shfl_xor_sync(0xffffffffu, z0, d);
        z1 += __shfl_xor_sync(0xffffffffu, z1, d);
      }
    }
    if (lane == 0) {
      o[k] = (prefactor * (s[0].y + s[3].y) - z0) / norm;
      o[k + 1] = (prefactor * (s[0].y - s[3].y) - z1) / norm;
    }
    k += 2;
  }
  if (do_ext && lane == 0) {
    o[k] = prefactor * (s[0].y + s[3].y) / norm;
    o[k + 1] = prefactor * (s[0].y - s[3].y) / norm;
    o[k + 2] = prefactor * (s[3].x - s[0].x) / norm;
  }
}

// One thread per (grain, theta): derivatives of (Qext, Qextpol, Qextcpol)
// with respect to (Re m, Im m, R_V, d) from the tangent amplitudes. S is
// linear in T, and T is holomorphic in m, so dS/d(Im m) = i dS/d(Re m); the
// normalisation 1/(pi R_V^2) adds -2 Q / R_V to the R_V derivative.
// dq[(job.out * 3 + k) * 4 + p]
__global__ void k_dq_epilogue(const TmxQJob *__restrict__ jobs, int njobs,
                              const TmxObsGrain *__restrict__ og,
                              const cplx *__restrict__ S,
                              const cplx *__restrict__ dSm,
                              const cplx *__restrict__ dSr,
                              const cplx *__restrict__ dSd,
                              double *__restrict__ dq) {
  const int u = blockIdx.x * blockDim.x + threadIdx.x;
  if (u >= njobs) {
    return;
  }
  const TmxQJob J = jobs[u];
  const TmxObsGrain G = og[J.grain];
  const double f = (2. * M_PI / G.k) / (M_PI * G.r_ev * G.r_ev);
  const cplx *s = S + J.s_main * 4;
  const double q[3] = {f * (s[0].y + s[3].y), f * (s[0].y - s[3].y),
                       f * (s[3].x - s[0].x)};
  const cplx *dm = dSm + J.s_main * 4;
  const cplx *dr = dSr + J.s_main * 4;
  const cplx *dd = dSd + J.s_main * 4;
  double *o = dq + J.out * 12;
  // Re m
  o[0 * 4 + 0] = f * (dm[0].y + dm[3].y);
  o[1 * 4 + 0] = f * (dm[0].y - dm[3].y);
  o[2 * 4 + 0] = f * (dm[3].x - dm[0].x);
  // Im m: Im(i z) = Re z, Re(i z) = -Im z
  o[0 * 4 + 1] = f * (dm[0].x + dm[3].x);
  o[1 * 4 + 1] = f * (dm[0].x - dm[3].x);
  o[2 * 4 + 1] = -f * (dm[3].y - dm[0].y);
  // R_V
  o[0 * 4 + 2] = f * (dr[0].y + dr[3].y) - 2. * q[0] / G.r_ev;
  o[1 * 4 + 2] = f * (dr[0].y - dr[3].y) - 2. * q[1] / G.r_ev;
  o[2 * 4 + 2] = f * (dr[3].x - dr[0].x) - 2. * q[2] / G.r_ev;
  // axis ratio
  o[0 * 4 + 3] = f * (dd[0].y + dd[3].y);
  o[1 * 4 + 3] = f * (dd[0].y - dd[3].y);
  o[2 * 4 + 3] = f * (dd[3].x - dd[0].x);
}

// one thread per (grain, theta_out, phi_out): the 4x4 matrix of
// ScatteringMatrixTask::execute from S, row major
__global__ void k_z_epilogue(int n, const cplx *__restrict__ S,
                             double *__restrict__ zout) {
  const int u = blockIdx.x * blockDim.x + threadIdx.x;
  if (u >= n) {
    return;
  }
  const cplx *s = S + (int64_t)u * 4;
  const cplx S0 = s[0], S1 = s[1], S2 = s[2], S3 = s[3];
  auto cj = [](cplx a) { return mkc(a.x, -a.y); };
  auto re_i = [](cplx a) { return -a.y; }; // Re(i a)
  double *Z = zout + (int64_t)u * 16;
  Z[0] = zsum(s, 1., 1., 1.);
  Z[1] = 0.5 * (cnorm2(S0) - cnorm2(S1) + cnorm2(S2) - cnorm2(S3));
  Z[2] = (csub(mkc(0., 0.), cadd(cmul(S0, cj(S1)), cmul(S3, cj(S2))))).x;
  Z[3] = re_i(csub(cmul(S0, cj(S1)), cmul(S3, cj(S2))));
  Z[4] = 0.5 * (cnorm2(S0) + cnorm2(S1) - cnorm2(S2) - cnorm2(S3));
  Z[5] = 0.5 * (cnorm2(S0) - cnorm2(S1) - cnorm2(S2) + cnorm2(S3));
  Z[6] = (cadd(mkc(-cmul(S0, cj(S1)).x, -cmul(S0, cj(S1)).y),
               cmul(S3, cj(S2)))).x;
  Z[7] = re_i(cadd(cmul(S0, cj(S1)), cmul(S3, cj(S2))));
  Z[8] = (csub(mkc(-cmul(S0, cj(S2)).x, -cmul(S0, cj(S2)).y),
               cmul(S3, cj(S1)))).x;
  Z[9] = (cadd(mkc(-cmul(S0, cj(S2)).x, -cmul(S0, cj(S2)).y),
               cmul(S3, cj(S1)))).x;
  Z[10] = cadd(cmul(S0, cj(S3)), cmul(S1, cj(S2))).x;
  Z[11] = -re_i(cadd(cmul(S0, cj(S3)), cmul(S2, cj(S1))));
  Z[12] = re_i(cadd(cmul(S2, cj(S0)), cmul(S3, cj(S1))));
  Z[13] = re_i(csub(cmul(S2, cj(S0)), cmul(S3, cj(S1))));
  Z[14] = -re_i(csub(cmul(S3, cj(S0)), cmul(S1, cj(S2))));
  Z[15] = csub(cmul(S3, cj(S0)), cmul(S1, cj(S2))).x;
}

// shape average: out[c][j] = sum_s w_s in[c][s][j] / sum_s w_s
__global__ void k_shape_avg(int ncells, int nshape, int nper,
                            const double *__restrict__ in,
                            const double *__restrict__ w,
                            double *__restrict__ out) {
  const int64_t u = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (u >= (int64_t)ncells * nper) {
    return;
  }
  const int64_t c = u / nper;
  const int j = (int)(u % nper);
  double acc = 0., norm = 0.;
  for (int s = 0; s < nshape; ++s) {
    acc += w[s] * in[(c * nshape + s) * nper + j];
    norm += w[s];
  }
  out[u] = acc * (1. / norm);
}

// --------------------------------------------------------- launchers -----

void tmx_launch_cg(int nmax, const int64_t *cg_off, double *cg, double *work,
                   int blocks, cudaStream_t stream) {
  k_cg<<<blocks, 128, 0, stream>>>(nmax, cg_off, cg, work);
}

// The attribute is the block's limit, not the launch's size: threads with
// contexts of their own launch the same kernel with different sizes, and one
// that lowered it between another's set and launch would fail that launch.
#define TMX_OBS_SMEM_MAX (227 * 1024)

template <int NT>
static void launch_orient(const TmxObsGrain *og, const int32_t *order,
                          const TmxOrientRange *rng, int nrng, int64_t nitems, int ncap,
                          const TmxMatSet &mats, int nmat, const double *coeffs,
                          int ncoef, const int64_t *cg_off, const double *cg,
                          int cg_nmax, int fold, cudaStream_t stream) {
  // t and S: rows of M + 1 <= ncap + 1 orders, padded to tiles
  const int rows = ncap + 1;
  const size_t smem = (size_t)4 * 2 * ((rows + 7) & ~7) * (8 * NT + 4) * sizeof(double);
  cudaFuncSetAttribute(k_orient<NT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       TMX_OBS_SMEM_MAX);
  k_orient<NT><<<dim3((unsigned)((nitems + 3) / 4), nmat), 128, smem, stream>>>(
      og, order, rng, nrng, nitems, rows, mats, coeffs, ncoef, cg_off, cg, cg_nmax, fold);
}

void tmx_launch_orient(const TmxObsGrain *og, const int32_t *order,
                       const TmxOrientRange *rng, int nrng, int64_t nitems, int ncap,
                       int chunk, const TmxMatSet &mats, int nmat,
                       const double *coeffs, int ncoef, const int64_t *cg_off,
                       const double *cg, int cg_nmax, int fold, cudaStream_t stream) {
  if (nitems <= 0) {
    return;
  }
  const auto run = [&](auto f) {
    f(og, order, rng, nrng, nitems, ncap, mats, nmat, coeffs, ncoef, cg_off, cg, cg_nmax,
      fold, stream);
  };
  run(chunk <= 2 ? launch_orient<1> : chunk <= 4 ? launch_orient<2> : launch_orient<4>);
}

void tmx_launch_wigner_cols(const TmxAngle *angles, int nangles, int nmax,
                            double *pi, double *tau, cudaStream_t stream) {
  const int64_t n = (int64_t)nangles * (nmax + 1);
  if (n <= 0) {
    return;
  }
  k_wigner_cols<<<(int)((n + 127) / 128), 128, 0, stream>>>(angles, nangles, nmax,
                                                           pi, tau);
}

template <int NT, int NTH>
static void launch_amp(const TmxAmpGroup *groups, const int32_t *ins,
                       const TmxAmpPair *pairs, const TmxAmpRange *rng, int nrng,
                       int64_t nitems, const TmxObsGrain *og, const TmxMatSet &mats,
                       int nmat, const double *wpi, const double *wtau, int wnmax,
                       double2 *x, int64_t xstride, int lcap, cudaStream_t stream) {
  constexpr int NA = 4 * NT, VS = (NA > 8) ? 18 : 10;
  const size_t smem = (size_t)lcap * (2 * NA * 2 * sizeof(double2) + 2 * VS * sizeof(double));
  cudaFuncSetAttribute(k_amp<NT, NTH>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       TMX_OBS_SMEM_MAX);
  k_amp<NT, NTH><<<dim3((unsigned)nitems, nmat), NTH, smem, stream>>>(
      groups, ins, pairs, rng, nrng, og, mats, wpi, wtau, wnmax, x, xstride, lcap);
}

void tmx_launch_amp(const TmxAmpGroup *groups, const int32_t *ins,
                    const TmxAmpPair *pairs, const TmxAmpRange *rng, int nrng,
                    int64_t nitems, const TmxObsGrain *og, const TmxMatSet &mats,
                    int nmat, const double *wpi, const double *wtau, int wnmax,
                    double2 *x, int64_t xstride, int lcap, int nin,
                    cudaStream_t stream) {
  if (nitems <= 0) {
    return;
  }
  // column tiles of four angles; blocks of more than 32 orders have enough
  // row tiles for eight warps
  const auto run = [&](auto f) {
    f(groups, ins, pairs, rng, nrng, nitems, og, mats, nmat, wpi, wtau, wnmax, x,
      xstride, lcap, stream);
  };
  if (lcap > 32) {
    run(nin <= 4 ? launch_amp<1, 256> : nin <= 8 ? launch_amp<2, 256> : launch_amp<4, 256>);
  } else {
    run(nin <= 4 ? launch_amp<1, 128> : nin <= 8 ? launch_amp<2, 128> : launch_amp<4, 128>);
  }
}

void tmx_launch_azimuth(const TmxAmpGroup *groups, int ngroups,
                        const TmxAmpPair *pairs, const TmxObsGrain *og,
                        const TmxMatSet &mats, int nmat, const double2 *phis,
                        const double2 *x, int64_t xstride, int nitem_max,
                        cudaStream_t stream) {
  if (ngroups <= 0) {
    return;
  }
  const int slices = std::max(1, std::min((nitem_max + 127) / 128, 1024));
  k_azimuth<<<dim3(ngroups, slices, nmat), 128, 0, stream>>>(groups, pairs, og, mats,
                                                             phis, x, xstride);
}

void tmx_launch_q_epilogue(const TmxQJob *jobs, int njobs, const TmxObsGrain *og,
                           const double2 *S, const double *wts, int nacc,
                           double *qout, int qstride, int do_abs, int do_ext,
                           cudaStream_t stream) {
  if (njobs <= 0) {
    return;
  }
  if (nacc > 0 && do_abs) {
    k_q_epilogue<true><<<(njobs + 3) / 4, 128, 0, stream>>>(
        jobs, njobs, og, S, wts, nacc, qout, qstride, do_abs, do_ext);
  } else {
    k_q_epilogue<false><<<(njobs + 127) / 128, 128, 0, stream>>>(
        jobs, njobs, og, S, wts, nacc, qout, qstride, do_abs, do_ext);
  }
}

void tmx_launch_dq_epilogue(const TmxQJob *jobs, int njobs,
                            const TmxObsGrain *og, const double2 *S,
                            const double2 *dSm, const double2 *dSr,
                            const double2 *dSd, double *dq, cudaStream_t stream) {
  if (njobs <= 0) {
    return;
  }
  k_dq_epilogue<<<(njobs + 127) / 128, 128, 0, stream>>>(jobs, njobs, og, S,
                                                         dSm, dSr, dSd, dq);
}

void tmx_launch_z_epilogue(int n, const double2 *S, double *zout,
                           cudaStream_t stream) {
  if (n <= 0) {
    return;
  }
  k_z_epilogue<<<(n + 127) / 128, 128, 0, stream>>>(n, S, zout);
}

void tmx_launch_shape_avg(int ncells, int nshape, int nper, const double *in,
                          const double *w, double *out, cudaStream_t stream) {
  const int64_t n = (int64_t)ncells * nper;
  if (n <= 0) {
    return;
  }
  k_shape_avg<<<(unsigned)((n + 255) / 256), 256, 0, stream>>>(ncells, nshape,
                                                               nper, in, w, out);
}

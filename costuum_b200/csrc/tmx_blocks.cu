// Block kernels: for one (grain, m, parity class) work item, assemble the
// class sub-matrices of Q and RgQ by quadrature, factor Q with partial
// pivoting in shared memory and solve T_c Q_c = -RgQ_c.
//
// Reference semantics (CosTuuM):
//   assembly  TMatrixM0Task::execute   src/TMatrixResource.hpp:601-709 (m=0)
//             TMatrixMAllTask::execute src/TMatrixResource.hpp:934-1100
//   inversion Matrix::plu_inverse      src/Matrix.hpp:261-384
//   T         T = -RgQ Q^-1            src/TMatrixResource.hpp:712-730
//
// Restructuring (same mathematics):
//  * Parity classes. Q_m has non-zero entries only where the row label
//    (i + n) % 2 equals the column label (m >= 1), and is block diagonal in i
//    for m = 0. Partial pivoting never picks a row of another class (those
//    entries are exact zeros) and elimination never mixes classes, so the
//    reference's LU of the full 2nb x 2nb block performs, entry for entry,
//    the LUs of the independent classes. Each class is one work item here.
//  * Assembly as a GEMM. Every entry is sum_g sum_{t<4} F_t(g, n1) W_t(g, n2)
//    with A-side vectors built from h_n1 = j + i y (or j alone for RgQ) and
//    B-side vectors built from j_n2(m k r); see below.
//  * T = -RgQ Q^-1 by two triangular solves on the LU factors instead of the
//    explicit inverse followed by a product.
#include <algorithm>
#include <type_traits>

#include "tmx_blocks_common.cuh"


// Build the A-side (F) and B-side (W) vectors of nodes [g0, g0 + G).
//   F1 = a d h, F2 = a dd h, F3 = a d dh, F4 = a (dd dh + n(n+1) drr/kr d h)
//   G1 = a d dj~, G2 = a (dd dj~ + drr/(m k r) n(n+1) d j~), G3 = a d j~,
//   G4 = a dd j~  (j~ = j_n(m k r), dj~ its derivative form)
//   alpha = w r^2, mu = m^2 / sin^2, beta = m w r^2 / sin
//   Q11: W = (k2mr a mu G1, k2mr a G2, -k2 a mu G3, -k2 a G4)
//   Q22: W = (k2 a mu G1, k2 a G2, -k2mr a mu G3, -k2mr a G4)
//   Q12: W = i (k2mr b G4, k2mr b G3, k2 b G2, k2 b G1)
//   Q21: W = i (k2 b G4, k2 b G3, k2mr b G2, k2mr b G1)
// This is the expansion of the J11, J12, J21, J22 terms of
// TMatrixResource.hpp:993-1097 into products of one n1 factor and one n2
// factor per node.
// A-side vectors (F^j, F^y) of row member a at node g, stored to f[t * ts].
// LEAN: without the factor a_n (the caller scales the finished entries by
// a_n1 a_n2) and, for m = 0, only the terms 1 and 3 that survive mu = 0.
// (an: a_n of the row, not used by LEAN)
template <bool LEAN = false>
__device__ __forceinline__ void a_side_row(double j, double dj, double y,
                                           double dy, double d, double dd,
                                           const double *s, int n, cplx *f,
                                           int ts, int m, double an = 1.) {
  const double nn = n * (n + 1.);
  const double q = nn * s[TMX_NS_DRR] * s[TMX_NS_KRINV] * d;
  if (LEAN) {
    if (m != 0) {
      f[0] = mkc(d * j, d * y);
      f[2 * ts] = mkc(d * dj, d * dy);
    }
    f[ts] = mkc(dd * j, dd * y);
    f[3 * ts] = mkc(dd * dj + q * j, dd * dy + q * y);
    return;
  }
  f[0] = mkc(an * d * j, an * d * y);
  f[ts] = mkc(an * dd * j, an * dd * y);
  f[2 * ts] = mkc(an * d * dj, an * d * dy);
  f[3 * ts] = mkc(an * (dd * dj + q * j), an * (dd * dy + q * y));
}

// B-side vectors of column member (ib, n) at one node for the rows of block
// index ia, stored to wr[t * ts]. LEAN as for a_side.
struct BSide {
  cplx G1, G2, G3, G4;
  double wr2, mu, beta;
};
template <bool LEAN>
__device__ __forceinline__ BSide b_side_node(int n, int m, cplx jm, cplx djm, double d,
                                             double dd, const double *s,
                                             double an = 1.) {
  BSide B;
  const double nn = n * (n + 1.);
  const cplx kmi = mkc(s[TMX_NS_KRMRINV_RE], s[TMX_NS_KRMRINV_IM]);
  B.G1 = cscale(djm, an * d);
  B.G2 = cscale(
      cadd(cscale(djm, dd), cscale(cmul(kmi, jm), s[TMX_NS_DRR] * nn * d)), an);
  B.G3 = cscale(jm, an * d);
  B.G4 = cscale(jm, an * dd);
  B.wr2 = s[TMX_NS_W] * s[TMX_NS_R2];
  B.mu = (double)(m * m) * s[TMX_NS_SIN2INV];
  B.beta = s[TMX_NS_SININV] * m * B.wr2;
  return B;
}
template <bool LEAN>
__device__ __forceinline__ void b_side_terms(const BSide &B, int ia, int ib, int m,
                                             double k2, cplx k2mr, cplx *wr, int ts) {
  if (ia == ib) {
    // diagonal-type block: Q11 (i = 0) or Q22 (i = 1)
    const cplx chi = (ia == 0) ? k2mr : mkc(k2, 0.);
    const cplx clo = (ia == 0) ? mkc(-k2, 0.) : mkc(-k2mr.x, -k2mr.y);
    if (!LEAN || m != 0) {
      wr[0] = cmul(chi, cscale(B.G1, B.wr2 * B.mu));
      wr[2 * ts] = cmul(clo, cscale(B.G3, B.wr2 * B.mu));
    }
    wr[ts] = cmul(chi, cscale(B.G2, B.wr2));
    wr[3 * ts] = cmul(clo, cscale(B.G4, B.wr2));
  } else {
    // off-diagonal block: Q12 (ia = 0, ib = 1) or Q21 (ia = 1, ib = 0)
    const cplx c1 = (ia == 0) ? k2mr : mkc(k2, 0.);
    const cplx c2 = (ia == 0) ? mkc(k2, 0.) : k2mr;
    const cplx ic1 = mkc(-c1.y * B.beta, c1.x * B.beta); // i c1 beta
    const cplx ic2 = mkc(-c2.y * B.beta, c2.x * B.beta);
    wr[0] = cmul(ic1, B.G4);
    wr[ts] = cmul(ic1, B.G3);
    wr[2 * ts] = cmul(ic2, B.G2);
    wr[3 * ts] = cmul(ic2, B.G1);
  }
}

// B-side vectors of a column member for each row group, stored to
// w[rg * gs + t * ts] (rg = 0 rows of block index D.iA, rg = 1 rows of D.iB).
template <bool LEAN = false>
__device__ __forceinline__ void b_side_row(const ClassDesc &D, int ib, int n,
                                           int m, cplx jm, cplx djm, double d,
                                           double dd, const double *s,
                                           int ngroups, double k2, cplx k2mr,
                                           cplx *w, int ts, int gs) {
  const BSide B = b_side_node<LEAN>(n, m, jm, djm, d, dd, s);
  for (int rg = 0; rg < ngroups; ++rg) {
    b_side_terms<LEAN>(B, (rg == 0) ? D.iA : D.iB, ib, m, k2, k2mr, w + rg * gs, ts);
  }
}

// zero A-side / B-side entries (padding and nodes past ngauss)
__device__ __forceinline__ void zero_side(cplx *f, int ts, int nt) {
  for (int t = 0; t < nt; ++t) {
    f[t * ts] = mkc(0., 0.);
  }
}

// ------------------------------------------------- warp-per-item variant --
//
// Classes of at most 16 members (nearly every item of grains up to order 32)
// are too small for a CTA: one warp owns one item from assembly to write-out
// and synchronises with __syncwarp only, so four independent items share a
// CTA. Assembly: lane (rt, ct) = (lane / 4, lane % 4) accumulates rows
// rt * TR .. rt * TR + TR - 1 and columns ct, ct + 4, .. of the class matrix
// over warp-private chunks of WG nodes. LU: lane r updates row r; the pivot
// column's maximum is a shuffle reduction (first maximum wins, as
// in Matrix::plu_inverse) and the factors stay in warp-private shared
// memory. Solve: lane r owns row r of -RgQ_c and runs both triangular solves
// on it against the factors, so no lane waits on another.

#ifndef TMX_WG
#define TMX_WG 4 // quadrature nodes per warp chunk (a multiple of 4)
#endif
// resident CTAs of four warps per SM the warp kernels are compiled for
// (register budget 65536 / (128 x MINB) per thread)
#ifndef TMX_WARP_DFMA_MINB
#define TMX_WARP_DFMA_MINB 4
#endif
#ifndef TMX_WARP_DMMA_MINB
#define TMX_WARP_DMMA_MINB 3
#endif

template <int NBM>
__host__ __device__ constexpr int warp_elems() {
  // chunk buffers F[WG][4][NBM] + W[2][WG][4][NBM]; the LU phase reuses them
  // for Q, RgQ ([NBM][NBM + 1] each), 1/U_jj and the pivot/gather indices
  return 12 * TMX_WG * NBM;
}

// Staging area of the next chunk's table rows (complex units): per node and
// class member one row of TMX_ROW doubles (the Bessel row j, j', y, y', j~,
// j~' and the Wigner pair d, d'; 80 bytes, so 16-byte reads of consecutive
// members hit distinct banks), and the node's scalar row (TMX_NS doubles).
#define TMX_ROW 10
template <int NBM>
__host__ __device__ constexpr int warp_stage_elems() {
  return TMX_WG * (NBM * TMX_ROW + TMX_NS) / 2;
}

// 16-byte asynchronous global -> shared copies (L2 only)
__device__ __forceinline__ void cp16(void *dst, const void *src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(src)
               : "memory");
}
__device__ __forceinline__ void cp_commit() {
  asm volatile("cp.async.commit_group;\n" ::: "memory");
}
__device__ __forceinline__ void cp_wait_all() {
  asm volatile("cp.async.wait_all;\n" ::: "memory");
}

// Copies of one item's table rows into the staging area. Each lane owns up
// to SL_MAX 16-byte pieces of the member rows (piece p < 4 of the Bessel row
// of member a, or p = 4: its Wigner pair) and one piece of the node scalars;
// their source addresses at node 0 and their per-node strides are set up
// once per item, so a chunk costs one add and one copy per piece and node.
// Rows start on 16-byte boundaries: table offsets are multiples of TMX_NQ
// (8) doubles, Wigner offsets of 2 and node-scalar offsets of TMX_NS (16).
template <int NBM>
struct StagePlan {
  static constexpr int SL_MAX = (NBM * 5 + 31) / 32;
  // TMX_WG nodes x TMX_NS / 2 pieces of node scalars, SS per lane
  static constexpr int SS = TMX_WG * (TMX_NS / 2) / 32;
  static_assert(SS * 32 == TMX_WG * (TMX_NS / 2), "node-scalar pieces per lane");
  const double *src[SL_MAX]; // piece at node 0
  int stride[SL_MAX];        // doubles per node
  int dst[SL_MAX];           // double offset in the stage (node 0); -1: none
  const double *ssrc[SS];    // node-scalar pieces (at chunk start 0)
  int sdst[SS];
  int sgl[SS];               // node of each piece within the chunk

  __device__ __forceinline__ void init(const ClassDesc &D, int N,
                                       const double *__restrict__ T,
                                       const double *__restrict__ S,
                                       const double *__restrict__ Wg,
                                       int lane) {
#pragma unroll
    for (int j = 0; j < SL_MAX; ++j) {
      const int q = lane + 32 * j;
      dst[j] = -1;
      src[j] = T;
      stride[j] = 0;
      if (q < D.nb * 5) {
        const int a = q / 5;
        const int p = q - 5 * a;
        int ia, n;
        member(D, a, ia, n);
        src[j] = (p < 4) ? T + (int64_t)(n - 1) * TMX_NQ + 2 * p
                         : Wg + (int64_t)(n - 1) * 2;
        stride[j] = (p < 4) ? N * TMX_NQ : 2 * N;
        dst[j] = a * TMX_ROW + 2 * p;
      }
    }
#pragma unroll
    for (int j = 0; j < SS; ++j) {
      const int q = lane + 32 * j;
      const int gl = q / (TMX_NS / 2);
      const int p = q - gl * (TMX_NS / 2);
      ssrc[j] = S + (int64_t)gl * TMX_NS + 2 * p;
      sdst[j] = TMX_WG * NBM * TMX_ROW + gl * TMX_NS + 2 * p;
      sgl[j] = gl;
    }
  }

  // copies of nodes [g0, g0 + TMX_WG) (one commit group per lane)
  __device__ __forceinline__ void issue(double *st, int g0, int ng) const {
#pragma unroll
    for (int j = 0; j < SL_MAX; ++j) {
      if (dst[j] >= 0) {
        const double *sp = src[j] + (int64_t)g0 * stride[j];
#pragma unroll
        for (int gl = 0; gl < TMX_WG; ++gl) {
          if (g0 + gl < ng) {
            cp16(st + dst[j] + gl * NBM * TMX_ROW, sp);
          }
          sp += stride[j];
        }
      }
    }
#pragma unroll
    for (int j = 0; j < SS; ++j) {
      if (g0 + sgl[j] < ng) {
        cp16(st + sdst[j], ssrc[j] + (int64_t)g0 * TMX_NS);
      }
    }
    cp_commit();
  }
};

// D += A B for one m8n8k4 FP64 tensor-core tile: lane l holds A[l / 4][l % 4],
// B[l % 4][l / 4] and D[l / 4][2 (l % 4) + {0, 1}]
__device__ __forceinline__ void dmma(double &d0, double &d1, double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, "
      "{%0, %1};\n"
      : "+d"(d0), "+d"(d1)
      : "d"(a), "d"(b));
}

// Complex products with their roundings spelled out (the compiler may contract
// either product of a sum, and large elongated grains amplify the last bit of
// a factor by many orders of magnitude): mul_xy fuses the x x and y x products,
// mul_xx the x x and x y ones, mul_yx the y y and x y ones. k_blocks_cta32,
// k_factor and k_solve form l = q / u with mul_xx and update with mul_xy; the warp
// kernels leave their products to the compiler, which contracts them alike. So
// the families for up to 64 members give a class the same T, bit for bit. The
// family for up to 128 (k_assemble<false>) applies the a_n to the node vectors
// instead of the finished entries: its T differs in the last bits, and so may a
// context whose dispatch table names it for smaller classes.
__device__ __forceinline__ cplx mul_xy(cplx a, cplx b) {
  return mkc(__fma_rn(a.x, b.x, -__dmul_rn(a.y, b.y)),
             __fma_rn(a.y, b.x, __dmul_rn(a.x, b.y)));
}
__device__ __forceinline__ cplx mul_xx(cplx a, cplx b) {
  return mkc(__fma_rn(a.x, b.x, -__dmul_rn(a.y, b.y)),
             __fma_rn(a.x, b.y, __dmul_rn(a.y, b.x)));
}
__device__ __forceinline__ cplx mul_yx(cplx a, cplx b) {
  return mkc(__fma_rn(-a.y, b.y, __dmul_rn(a.x, b.x)),
             __fma_rn(a.x, b.y, __dmul_rn(a.y, b.x)));
}

// ------------------------------------------ LU and solves in registers --
//
// Row r of a class matrix lives in the registers of the C lanes
// [C r, C r + C) of a warp: lane c of the group holds the columns
// k = c + C t (t < NBM / C). Both routines perform the operations of the
// one-row-per-lane versions in the same order.

// Pivot of one elimination step: the candidate with the largest key (the
// bits of |Q_ri| with the top bit set, which order like the non-negative
// doubles; 0 for lanes that are no candidate), ties to the smallest position.
__device__ __forceinline__ void warp_argmax(unsigned long long key, int pos,
                                            int &best_pos, int &best_lane) {
  const unsigned hi = (unsigned)(key >> 32), lo = (unsigned)key;
  const unsigned mh = __reduce_max_sync(0xffffffffu, hi);
  const unsigned ml = __reduce_max_sync(0xffffffffu, (hi == mh) ? lo : 0u);
  const bool top = (hi == mh) && (lo == ml) && key != 0ull;
  const unsigned mp = __reduce_min_sync(0xffffffffu, top ? (unsigned)pos : 0xffffffffu);
  const unsigned bal = __ballot_sync(0xffffffffu, top && (unsigned)pos == mp);
  best_pos = (int)mp;
  best_lane = __ffs(bal) - 1;
}

// Pivot of one elimination step over the lanes' candidates c (have: the lane has
// one): the first position with the largest |c|, as warp_argmax finds it from
// hypot. |c|^2 decides unless another candidate comes within rounding of the
// largest one (or the squares leave the range of doubles): then the hypots do.
// Returns whether the pivot is non-zero.
__device__ __forceinline__ bool warp_pivot(cplx c, bool have, int pos, int &best_pos,
                                           int &best_lane) {
  double s = have ? fma(c.x, c.x, c.y * c.y) : 0.;
  s = (s >= 0.) ? s : 0.; // (NaN is no candidate)
  const unsigned long long top = 1ull << 63;
  warp_argmax(have ? (unsigned long long)__double_as_longlong(s) | top : 0ull, pos,
              best_pos, best_lane);
  const double best = __shfl_sync(0xffffffffu, s, best_lane);
  const bool close = have && s >= best * (1. - 0x1p-40);
  const bool odd = __popc(__ballot_sync(0xffffffffu, close)) != 1;
  if (odd || !(best > 0x1p-900 && best < 0x1p900)) {
    double av = have ? cabs_dev(c) : 0.;
    av = (av >= 0.) ? av : 0.;
    warp_argmax(have ? (unsigned long long)__double_as_longlong(av) | top : 0ull, pos,
                best_pos, best_lane);
    return __shfl_sync(0xffffffffu, av, best_lane) > 0.;
  }
  return true;
}

// In-place LU with partial pivoting of the nb x nb matrix Q (row stride LD,
// shared memory) by one warp: the pivot of step i is the first row (by
// position) at or below i with the largest |Q_ri| (Matrix::plu_inverse,
// src/Matrix.hpp:261-384); rows stay in their lanes and carry a position.
// prow: NBM complex of scratch. Returns true if a pivot was zero.
template <int NBM, int C>
__device__ __forceinline__ bool lu_rows(cplx *Qm, int LD, cplx *prow, int *piv,
                                        int nb, int lane) {
  constexpr int NT = NBM / C;
  const int row = lane / C;
  const int c = lane % C;
  cplx q[NT];
#pragma unroll
  for (int t = 0; t < NT; ++t) {
    const int k = c + C * t;
    q[t] = (row < nb && k < nb) ? Qm[row * LD + k] : mkc(0., 0.);
  }
  int pos = row;
  bool singular = false;
#pragma unroll
  for (int i = 0; i < NBM; ++i) {
    if (i >= nb) {
      break;
    }
    const bool own = (c == i % C);
    double av = 0.;
    unsigned long long key = 0ull;
    if (own && row < nb && pos >= i) {
      av = cabs_dev(q[i / C]);
      key = (unsigned long long)__double_as_longlong(av) | (1ull << 63);
    }
    int bi, wl;
    warp_argmax(key, pos, bi, wl);
    const double best = __shfl_sync(0xffffffffu, av, wl);
    singular = singular || !(best > 0.);
    if (lane == 0) {
      piv[i] = bi;
    }
    const int wrow = wl / C;
    if (pos == i) {
      pos = bi;
    }
    if (row == wrow) {
      pos = i;
#pragma unroll
      for (int t = 0; t < NT; ++t) {
        const int k = c + C * t;
        if (k >= i && k < nb) {
          prow[k] = q[t];
        }
      }
    }
    __syncwarp();
    const bool elim = row < nb && pos > i;
    cplx l = mkc(0., 0.);
    if (elim && own) {
      const cplx pinv = cinv_lu(prow[i]);
      l = cmul(q[i / C], pinv);
      q[i / C] = l;
    }
    l.x = __shfl_sync(0xffffffffu, l.x, i % C, C);
    l.y = __shfl_sync(0xffffffffu, l.y, i % C, C);
    if (elim) {
#pragma unroll
      for (int t = 0; t < NT; ++t) {
        const int k = c + C * t;
        if (k > i && k < nb) {
          q[t] = csub(q[t], cmul(l, prow[k]));
        }
      }
    }
    __syncwarp();
  }
  if (row < nb) {
#pragma unroll
    for (int t = 0; t < NT; ++t) {
      const int k = c + C * t;
      if (k < nb) {
        Qm[pos * LD + k] = q[t];
      }
    }
  }
  return singular;
}

template <int TR, int TC, int MINB, bool MMA>
__global__ void __launch_bounds__(128, MINB)
    k_blocks_warp(TmxBlockArgs A) {
  constexpr int NBM = MMA ? 16 : ((8 * TR > 4 * TC) ? 8 * TR : 4 * TC);
  // row padding unit of the class rows: a tensor row tile of 8 holds one
  // row group only
  constexpr int PR = MMA ? 8 : TR;
  constexpr int LD = NBM + 1;
  static_assert(2 * NBM * LD + 2 * NBM <= warp_elems<NBM>(), "warp smem");
  extern __shared__ __align__(16) unsigned char tmx_wsmem[];
  const int lane = threadIdx.x & 31;
  const int wib = threadIdx.x >> 5;
  cplx *base = reinterpret_cast<cplx *>(tmx_wsmem) + wib * warp_elems<NBM>();
  cplx *Fs = base;                      // [WG][4][NBM]
  cplx *Ws = Fs + TMX_WG * 4 * NBM;     // [2][WG][4][NBM]
  cplx *Qm = base;                      // [NBM][LD]  (after the assembly)
  cplx *Rm = Qm + NBM * LD;             // [NBM][LD]
  cplx *uinv = Rm + NBM * LD;           // [NBM]
  int *perm = reinterpret_cast<int *>(uinv + NBM); // [NBM]
  int *piv = perm + NBM;                           // [NBM]
  double *stg = reinterpret_cast<double *>(
      reinterpret_cast<cplx *>(tmx_wsmem) + 4 * warp_elems<NBM>() +
      wib * warp_stage_elems<NBM>());
  const double *stgS = stg + TMX_WG * NBM * TMX_ROW;
  const int rt = lane >> 2;
  const int ct = lane & 3;
  const int ilo = A.range ? A.range[0] : 0;
  const int ihi = A.range ? min(A.range[1], A.nitems) : A.nitems;
  for (int it = ilo + blockIdx.x * 4 + wib; it < ihi; it += gridDim.x * 4) {
    const TmxItem item = A.items[it];
    const TmxSlot sl = A.slots[item.slot];
    const TmxGrain Gr = A.grains[sl.grain];
    const int N = sl.nmax;
    const int ng = sl.ngauss;
    const int m = item.m;
    const ClassDesc D = describe<PR>(N, m, item.cls);
    const int nb = D.nb;
    if (nb <= 0) {
      continue;
    }
    if (nb > NBM || D.NRp > NBM) {
      if (lane == 0) {
        atomicOr(&A.status[sl.grain], TMX_ST_TOO_LARGE);
      }
      continue;
    }
    const double *T = A.tab + sl.tab;
    const double *S = A.nsc + sl.nsc;
    const double *Wg = A.wig + A.wig_off[sl.wig_n] + (int64_t)m * ng * N * 2;
    const double k2 = Gr.k * Gr.k;
    const cplx k2mr = mkc(Gr.mr * k2, Gr.mi * k2);
    const int ngroups = (D.R1 > 0 && m > 0) ? 2 : 1;

    // ---------------------------------------------------------- assembly
    // DFMA path: aj/ay[TR][TC]; tensor path: acc[row tile][col tile][jr, ji,
    // yr, yi] as m8n8 accumulator fragments
    double aj[TR][TC][2], ay[TR][TC][2];
    double acc[2][2][4][2];
#pragma unroll
    for (int r = 0; r < TR; ++r) {
#pragma unroll
      for (int c = 0; c < TC; ++c) {
        aj[r][c][0] = aj[r][c][1] = ay[r][c][0] = ay[r][c][1] = 0.;
      }
    }
#pragma unroll
    for (int r = 0; r < 2; ++r) {
#pragma unroll
      for (int c = 0; c < 2; ++c) {
#pragma unroll
        for (int p = 0; p < 4; ++p) {
          acc[r][c][p][0] = acc[r][c][p][1] = 0.;
        }
      }
    }
    // rows are padded per group to a multiple of TR (describe<TR>), so the
    // TR rows of a lane share one row group and one set of B-side vectors
    const int rgl = (rt * TR < D.R0p) ? 0 : 1;
    // the table rows of each chunk are staged in shared memory while the
    // previous chunk is contracted
    StagePlan<NBM> plan;
    plan.init(D, N, T, S, Wg, lane);
    plan.issue(stg, 0, ng);
    for (int g0 = 0; g0 < ng; g0 += TMX_WG) {
      cp_wait_all();
      __syncwarp();
      // slots (node gl, row or column) = (u / NBM, u % NBM): TMX_WG NBM / 32
      // per lane on each side, unrolled so that their shared-memory reads and
      // arithmetic interleave
      constexpr int NIT = TMX_WG * NBM / 32;
      static_assert(NIT * 32 == TMX_WG * NBM, "build slots");
#pragma unroll
      for (int j = 0; j < NIT; ++j) {
        const int u = lane + 32 * j;
        const int gl = u / NBM;
        const int pr = u % NBM;
        if (pr >= D.NRp) {
          continue;
        }
        const int a = padded_member(D, pr);
        cplx *fp = Fs + gl * 4 * NBM + pr;
        if (a >= 0 && g0 + gl < ng) {
          int ia, n;
          member(D, a, ia, n);
          const double *r = stg + (gl * NBM + a) * TMX_ROW;
          const double2 jd = *reinterpret_cast<const double2 *>(r + TMX_Q_J);
          const double2 yd = *reinterpret_cast<const double2 *>(r + TMX_Q_Y);
          const double2 wd = *reinterpret_cast<const double2 *>(r + TMX_NQ);
          a_side_row<true>(jd.x, jd.y, yd.x, yd.y, wd.x, wd.y, stgS + gl * TMX_NS,
                           n, fp, NBM, m);
        } else {
          zero_side(fp, NBM, 4);
        }
      }
#pragma unroll
      for (int j = 0; j < NIT; ++j) {
        const int u = lane + 32 * j;
        const int gl = u / NBM;
        const int b = u % NBM;
        if (b >= nb) {
          continue;
        }
        cplx *wp = Ws + gl * 4 * NBM + b;
        if (g0 + gl < ng) {
          int ib, n;
          member(D, b, ib, n);
          const double *r = stg + (gl * NBM + b) * TMX_ROW;
          const double2 jm = *reinterpret_cast<const double2 *>(r + TMX_Q_JM_RE);
          const double2 djm = *reinterpret_cast<const double2 *>(r + TMX_Q_DJM_RE);
          const double2 wd = *reinterpret_cast<const double2 *>(r + TMX_NQ);
          b_side_row<true>(D, ib, n, m, jm, djm, wd.x, wd.y, stgS + gl * TMX_NS,
                           ngroups, k2, k2mr, wp, NBM, TMX_WG * 4 * NBM);
        } else {
          for (int q = 0; q < ngroups; ++q) {
            zero_side(wp + q * TMX_WG * 4 * NBM, NBM, 4);
          }
        }
      }
      __syncwarp();
      if (g0 + TMX_WG < ng) {
        plan.issue(stg, g0 + TMX_WG, ng);
      }
      const int gmax = min(TMX_WG, ng - g0);
      if constexpr (MMA) {
        // K slices of 4: the four terms of one node (m >= 1), or terms 1 and
        // 3 of two nodes (m = 0, where terms 0 and 2 vanish)
        // padded row tile rti holds row group (rti * 8 < R0p ? 0 : 1) only
        const int q = lane & 3;
        const int rr = lane >> 2;
        const int nrt = D.NRp >> 3;
        const int nct = (nb + 7) >> 3;
        const int nsl = (m == 0) ? (gmax + 1) >> 1 : gmax;
        for (int sx = 0; sx < nsl; ++sx) {
          const int gl = (m == 0) ? 2 * sx + (q >> 1) : sx;
          const int t = (m == 0) ? 1 + 2 * (q & 1) : q;
#pragma unroll
          for (int rti = 0; rti < 2; ++rti) {
            if (rti < nrt) {
              const cplx f = Fs[(gl * 4 + t) * NBM + rti * 8 + rr];
              const int g = (rti * 8 < D.R0p) ? 0 : 1;
#pragma unroll
              for (int cti = 0; cti < 2; ++cti) {
                if (cti < nct) {
                  const int col = cti * 8 + rr;
                  const cplx w = (col < nb)
                      ? Ws[((g * TMX_WG + gl) * 4 + t) * NBM + col]
                      : mkc(0., 0.);
                  double *a4 = &acc[rti][cti][0][0];
                  dmma(a4[0], a4[1], f.x, w.x); // jr
                  dmma(a4[2], a4[3], f.x, w.y); // ji
                  dmma(a4[4], a4[5], f.y, w.x); // yr
                  dmma(a4[6], a4[7], f.y, w.y); // yi
                }
              }
            }
          }
        }
      } else {
        // one term t of node gl; the terms of a node are unrolled (t = 1, 3
        // for m = 0, where mu = 0 removes t = 0, 2) so their reads overlap
        auto term = [&](int gl, int t) {
          const cplx *fr = Fs + (gl * 4 + t) * NBM + rt * TR;
          const cplx *wr = Ws + (rgl * TMX_WG * 4 + gl * 4 + t) * NBM + ct;
          cplx w[TC];
#pragma unroll
          for (int c = 0; c < TC; ++c) {
            w[c] = wr[4 * c];
          }
#pragma unroll
          for (int r = 0; r < TR; ++r) {
            const cplx f = fr[r];
#pragma unroll
            for (int c = 0; c < TC; ++c) {
              aj[r][c][0] = fma(f.x, w[c].x, aj[r][c][0]);
              aj[r][c][1] = fma(f.x, w[c].y, aj[r][c][1]);
              ay[r][c][0] = fma(f.y, w[c].x, ay[r][c][0]);
              ay[r][c][1] = fma(f.y, w[c].y, ay[r][c][1]);
            }
          }
        };
        if (m == 0) {
          for (int gl = 0; gl < gmax; ++gl) {
            term(gl, 1);
            term(gl, 3);
          }
        } else {
          for (int gl = 0; gl < gmax; ++gl) {
#pragma unroll
            for (int t = 0; t < 4; ++t) {
              term(gl, t);
            }
          }
        }
      }
    }
    __syncwarp();
    // a_n of each member once per item (in the 1/U_jj slots, free until the
    // LU); entry (a, b) is scaled by a_n(n_a) a_n(n_b)
    double *an_s = reinterpret_cast<double *>(uinv);
    if (lane < nb) {
      int ia, na;
      member(D, lane, ia, na);
      an_s[lane] = a_n(na);
    }
    __syncwarp();
    // Q = G^j + i G^y, RgQ = G^j, into the (reused) chunk buffers
    if constexpr (MMA) {
      const int rr = lane >> 2;
      const int q = lane & 3;
#pragma unroll
      for (int rti = 0; rti < 2; ++rti) {
#pragma unroll
        for (int cti = 0; cti < 2; ++cti) {
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const int a = padded_member(D, rti * 8 + rr);
            const int b = cti * 8 + 2 * q + i;
            if (a >= 0 && b < nb) {
              const double sc = an_s[a] * an_s[b];
              const double jr = acc[rti][cti][0][i], ji = acc[rti][cti][1][i];
              const double yr = acc[rti][cti][2][i], yi = acc[rti][cti][3][i];
              Qm[a * LD + b] = mkc((jr - yi) * sc, (ji + yr) * sc);
              Rm[a * LD + b] = mkc(jr * sc, ji * sc);
            }
          }
        }
      }
    } else {
#pragma unroll
      for (int r = 0; r < TR; ++r) {
        const int a = padded_member(D, rt * TR + r);
#pragma unroll
        for (int c = 0; c < TC; ++c) {
          const int b = ct + 4 * c;
          if (a >= 0 && b < nb) {
            const double sc = an_s[a] * an_s[b];
            Qm[a * LD + b] = mkc((aj[r][c][0] - ay[r][c][1]) * sc,
                                 (aj[r][c][1] + ay[r][c][0]) * sc);
            Rm[a * LD + b] = mkc(aj[r][c][0] * sc, aj[r][c][1] * sc);
          }
        }
      }
    }
    __syncwarp();

    // ---------------------------------------------------------------- LU
    // in registers, 32 / NBM lanes per row; the pivot row goes through uinv
    constexpr int CL = 32 / NBM;
    const bool singular = lu_rows<NBM, CL>(Qm, LD, uinv, piv, nb, lane);
    __syncwarp();
    if (lane < nb) {
      uinv[lane] = cinv_lu(Qm[lane * LD + lane]);
    }
    if (lane == 0) {
      // column exchanges of Matrix::plu_inverse step 4, as a gather index
      for (int j = 0; j < nb; ++j) {
        perm[j] = j;
      }
      for (int j = nb - 1; j >= 0; --j) {
        const int p = piv[j];
        const int t = perm[j];
        perm[j] = perm[p];
        perm[p] = t;
      }
      if (singular) {
        atomicOr(&A.status[sl.grain], TMX_ST_SINGULAR);
      }
    }
    __syncwarp();
    if (A.lu) {
      cplx *Ls = A.lu + item.scratch;
      for (int u = lane; u < nb * nb; u += 32) {
        Ls[u] = Qm[(u / nb) * LD + (u % nb)];
      }
      int *ps = reinterpret_cast<int *>(Ls + (int64_t)nb * nb);
      for (int j = lane; j < nb; j += 32) {
        ps[j] = perm[j];
      }
    }

    // ------------------------------------------ solve T_c Q_c = -RgQ_c
    solve_rows<NBM, CL>(Rm, Qm, LD, uinv, nb, lane / CL, lane % CL);
    __syncwarp();
    // write out: T_c[a][b] = Y[a][perm[b]]
    if (sl.tout < 0) {
      if (lane < nb) {
        int ia, na;
        member(D, lane, ia, na);
        A.diag[sl.diag + ia * N + (na - 1)] = Rm[lane * LD + perm[lane]];
      }
    } else {
      cplx *Tb = A.tout + sl.tout + block_offset(N, m);
      const int w2 = 2 * D.nbb;
      for (int u = lane; u < nb * nb; u += 32) {
        const int a = u / nb;
        const int b = u - a * nb;
        int ia, na, ib, nbn;
        member(D, a, ia, na);
        member(D, b, ib, nbn);
        const int rowi = ia * D.nbb + (na - D.nmin);
        const int col = ib * D.nbb + (nbn - D.nmin);
        Tb[(int64_t)rowi * w2 + col] = Rm[a * LD + perm[b]];
      }
    }
    __syncwarp();
  }
}

template <int TR, int TC, int MINB, bool MMA>
static void launch_warp_variant(const TmxBlockArgs &a, cudaStream_t stream) {
  constexpr int NBM = MMA ? 16 : ((8 * TR > 4 * TC) ? 8 * TR : 4 * TC);
  const size_t smem =
      (size_t)4 * (warp_elems<NBM>() + warp_stage_elems<NBM>()) * sizeof(cplx);
  cudaFuncSetAttribute(k_blocks_warp<TR, TC, MINB, MMA>,
                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  // one item per warp: CTAs retire after one item, so that launches of the
  // high-priority order loop get SMs between them (a grid of long-lived
  // CTAs looping over items held the SMs for a whole round)
  int blocks = (int)std::max<int64_t>(1, ((int64_t)a.nitems + 3) / 4);
  if (a.max_ctas > 0) {
    blocks = std::min(blocks, a.max_ctas);
  }
  k_blocks_warp<TR, TC, MINB, MMA><<<blocks, 128, smem, stream>>>(a);
}

// ------------------------------------------ four warps per item (<= 32) --
//
// Classes of 17..32 members: one CTA of four warps per item.
// Assembly: chunks of TMX_WG32 nodes; thread t builds padded row and column
// t % 32 of node t / 32 from staged table rows (copied with cp.async while the
// previous chunk is contracted), then the warps share the 8 x 8 tiles (rows
// padded per group, so that a tile has one set of W) evenly on the FP64 tensor
// pipe, K = (node, term) ascending.
// LU: lane r of every warp holds row r of the columns w, w + 4, .. of its warp
// w in registers. Per step the owner of the pivot column has put it into
// shared memory; each warp finds the pivot itself (lanes in parallel: |q|,
// 1 / q), takes the pivot row by shuffles and updates its columns, the owner
// of the next column first: one barrier per step, no row exchanges.
// Solve: four lanes per row, in registers.
// Measured (B200): 80 items of 17..20 members alone on the chip 61 -> 40 us, 3018
// items of 17..32 members, 32..100 nodes, 0.74 -> 0.62 ms, against table rows
// loaded in the build, tiles split by column and the LU on warp 0. Bound by
// latency at 12 warps per SM (issue slots 42 %, FP64 and DMMA pipes together
// 52 % busy). 166 registers and three CTAs: at 128 registers (four CTAs) the
// contraction spills, 49 us and 0.61 ms; eight warps per item 35 us and 0.68 ms.

#define TMX_WG32 4

struct Cta32 {
  static constexpr int NBM = 32, LD = NBM + 1, LDK = NBM + 2;
  // F[4 WG][LDK], W[2][4 WG][LDK] (rows padded by two: the four terms and two
  // members that eight lanes read fall into distinct banks), then the staged
  // rows; or Q, RgQ [32][33] and 1 / U_jj
  static constexpr int CHUNK = 12 * TMX_WG32 * LDK;
  static constexpr int STAGE = TMX_WG32 * (NBM * TMX_ROW + TMX_NS) / 2;
  static constexpr int SOLVE = 2 * NBM * LD + NBM;
  static constexpr int ELEMS = CHUNK + STAGE > SOLVE ? CHUNK + STAGE : SOLVE;
};

__global__ void __launch_bounds__(128, 3) k_blocks_cta32(TmxBlockArgs A) {
  constexpr int NBM = Cta32::NBM, LD = Cta32::LD, LDK = Cta32::LDK, WG = TMX_WG32;
  constexpr int NTILE = 4; // tiles per warp
  extern __shared__ __align__(16) unsigned char tmx_c32smem[];
  __shared__ cplx colbuf[2][NBM];
  __shared__ int at[NBM];      // row at a position
  __shared__ double an_s[NBM]; // a_n of the members
  cplx *base = reinterpret_cast<cplx *>(tmx_c32smem);
  cplx *Fs = base;
  cplx *Ws = Fs + 4 * WG * LDK;
  double *stg = reinterpret_cast<double *>(base + Cta32::CHUNK);
  const double *stgS = stg + WG * NBM * TMX_ROW;
  cplx *Qm = base; // (after the assembly)
  cplx *Rm = Qm + NBM * LD;
  cplx *uinv = Rm + NBM * LD;
  const int tid = threadIdx.x;
  const int lane = tid & 31;
  const int wib = tid >> 5;
  const int q = lane & 3;
  const int rr = lane >> 2;
  const int ilo = A.range ? A.range[0] : 0;
  const int ihi = A.range ? min(A.range[1], A.nitems) : A.nitems;
  for (int it = ilo + blockIdx.x; it < ihi; it += gridDim.x) {
    const TmxItem item = A.items[it];
    const TmxSlot sl = A.slots[item.slot];
    const int N = sl.nmax;
    const int ng = sl.ngauss;
    const int m = item.m;
    const ClassDesc D = describe<8>(N, m, item.cls);
    const int nb = D.nb;
    if (nb <= 0) {
      continue;
    }
    if (nb > NBM || D.NRp > NBM) {
      if (tid == 0) {
        atomicOr(&A.status[sl.grain], TMX_ST_TOO_LARGE);
      }
      continue;
    }
    const TmxGrain Gr = A.grains[sl.grain];
    const double *T = A.tab + sl.tab;
    const double *S = A.nsc + sl.nsc;
    const double *Wg = A.wig + A.wig_off[sl.wig_n] + (int64_t)m * ng * N * 2;
    const double k2 = Gr.k * Gr.k;
    const cplx k2mr = mkc(Gr.mr * k2, Gr.mi * k2);
    const int ngroups = (D.R1 > 0 && m > 0) ? 2 : 1;
    const int nt = (m == 0) ? 2 : 4; // terms per node
    // this thread's 16-byte pieces of a node's rows (5 per member)
    const double *src[2];
    int stride[2], dst[2];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int p = tid + 128 * j;
      const int a = p / 5, piece = p - 5 * a;
      int ia, n;
      member(D, a, ia, n);
      const bool have = a < nb;
      n = have ? n : 1;
      src[j] = (piece < 4) ? T + (int64_t)(n - 1) * TMX_NQ + 2 * piece
                           : Wg + (int64_t)(n - 1) * 2;
      stride[j] = (piece < 4) ? N * TMX_NQ : 2 * N;
      dst[j] = have ? a * TMX_ROW + 2 * piece : -1;
    }
    const auto issue = [&](int g0) {
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        if (dst[j] >= 0) {
          const double *sp = src[j] + (int64_t)g0 * stride[j];
#pragma unroll
          for (int gl = 0; gl < WG; ++gl) {
            if (g0 + gl < ng) {
              cp16(stg + gl * NBM * TMX_ROW + dst[j], sp);
            }
            sp += stride[j];
          }
        }
      }
      if (tid < WG * (TMX_NS / 2) && g0 + tid / (TMX_NS / 2) < ng) {
        cp16(stg + WG * NBM * TMX_ROW + 2 * tid, S + (int64_t)g0 * TMX_NS + 2 * tid);
      }
      cp_commit();
    };
    issue(0);
    // this thread's padded row and its column of node gl
    const int gl = wib;
    const int ra = (lane < D.NRp) ? padded_member(D, lane) : -1;
    const bool wcol = (lane & ~7) < nb;
    int ri, rn, ci, cn;
    member(D, max(ra, 0), ri, rn);
    member(D, lane, ci, cn);
    if (tid < nb) {
      an_s[tid] = a_n(cn);
    }
    // this warp's tiles
    const int nct = (nb + 7) >> 3;
    const int ntl = (D.NRp >> 3) * nct;
    int fo[NTILE], wo[NTILE];
    double acc[NTILE][4][2];
#pragma unroll
    for (int i = 0; i < NTILE; ++i) {
      const int t = wib + 4 * i;
      const int row = (t / nct) * 8;
      fo[i] = q * LDK + row + rr;
      wo[i] = ((row < D.R0p ? 0 : 4 * WG) + q) * LDK + (t % nct) * 8 + rr;
#pragma unroll
      for (int p = 0; p < 4; ++p) {
        acc[i][p][0] = acc[i][p][1] = 0.;
      }
    }
    for (int g0 = 0; g0 < ng; g0 += WG) {
      cp_wait_all();
      __syncthreads(); // the chunk's rows are there; F and W are free
      const bool live = g0 + gl < ng;
      const double *ns = stgS + gl * TMX_NS;
      if (lane < D.NRp) {
        cplx v[4] = {mkc(0., 0.), mkc(0., 0.), mkc(0., 0.), mkc(0., 0.)};
        if (live && ra >= 0) {
          const double *r = stg + (gl * NBM + ra) * TMX_ROW;
          const double2 jd = *reinterpret_cast<const double2 *>(r + TMX_Q_J);
          const double2 yd = *reinterpret_cast<const double2 *>(r + TMX_Q_Y);
          const double2 wd = *reinterpret_cast<const double2 *>(r + TMX_NQ);
          a_side_row<true>(jd.x, jd.y, yd.x, yd.y, wd.x, wd.y, ns, rn, v, 1, m);
        }
        cplx *o = Fs + gl * nt * LDK + lane;
        if (m == 0) {
          o[0] = v[1];
          o[LDK] = v[3];
        } else {
          o[0] = v[0];
          o[LDK] = v[1];
          o[2 * LDK] = v[2];
          o[3 * LDK] = v[3];
        }
      }
      if (wcol) {
        BSide B = {};
        const bool have = live && lane < nb;
        if (have) {
          const double *r = stg + (gl * NBM + lane) * TMX_ROW;
          const double2 jm = *reinterpret_cast<const double2 *>(r + TMX_Q_JM_RE);
          const double2 djm = *reinterpret_cast<const double2 *>(r + TMX_Q_DJM_RE);
          const double2 wd = *reinterpret_cast<const double2 *>(r + TMX_NQ);
          B = b_side_node<true>(cn, m, jm, djm, wd.x, wd.y, ns);
        }
        for (int g = 0; g < ngroups; ++g) {
          cplx v[4] = {mkc(0., 0.), mkc(0., 0.), mkc(0., 0.), mkc(0., 0.)};
          if (have) {
            b_side_terms<true>(B, (g == 0) ? D.iA : D.iB, ci, m, k2, k2mr, v, 1);
          }
          cplx *o = Ws + (g * 4 * WG + gl * nt) * LDK + lane;
          if (m == 0) {
            o[0] = v[1];
            o[LDK] = v[3];
          } else {
            o[0] = v[0];
            o[LDK] = v[1];
            o[2 * LDK] = v[2];
            o[3 * LDK] = v[3];
          }
        }
      }
      __syncthreads();
      if (g0 + WG < ng) {
        issue(g0 + WG);
      }
      const int kmax = min(WG, ng - g0) * nt;
      for (int k0 = 0; k0 < kmax; k0 += 4) {
#pragma unroll
        for (int i = 0; i < NTILE; ++i) {
          if (wib + 4 * i < ntl) {
            const cplx f = Fs[fo[i] + k0 * LDK];
            const cplx w = Ws[wo[i] + k0 * LDK];
            dmma(acc[i][0][0], acc[i][0][1], f.x, w.x); // jr
            dmma(acc[i][1][0], acc[i][1][1], f.x, w.y); // ji
            dmma(acc[i][2][0], acc[i][2][1], f.y, w.x); // yr
            dmma(acc[i][3][0], acc[i][3][1], f.y, w.y); // yi
          }
        }
      }
    }
    __syncthreads();
    // Q = G^j + i G^y, RgQ = G^j (times a_n1 a_n2), into the chunk buffers
#pragma unroll
    for (int i = 0; i < NTILE; ++i) {
      const int t = wib + 4 * i;
      const int a = (t < ntl) ? padded_member(D, (t / nct) * 8 + rr) : -1;
      if (a >= 0) {
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int b = (t % nct) * 8 + 2 * q + e;
          if (b < nb) {
            const double sc = an_s[a] * an_s[b];
            const double jr = acc[i][0][e], ji = acc[i][1][e];
            const double yr = acc[i][2][e], yi = acc[i][3][e];
            Qm[a * LD + b] = mkc((jr - yi) * sc, (ji + yr) * sc);
            Rm[a * LD + b] = mkc(jr * sc, ji * sc);
          }
        }
      }
    }
    __syncthreads();
    // ---------------------------------------------------------------- LU
    cplx x[NBM / 4]; // row `lane`, columns wib + 4 t
    bool singular = false;
    int pos = lane;
#pragma unroll
    for (int t = 0; t < NBM / 4; ++t) {
      const int k = wib + 4 * t;
      x[t] = (lane < nb && k < nb) ? Qm[lane * LD + k] : mkc(0., 0.);
    }
    if (wib == 0) {
      colbuf[0][lane] = x[0];
    }
    __syncthreads();
    for (int i = 0; i < nb; ++i) {
      const cplx c = colbuf[i & 1][lane];
      cplx pinv = cinv_lu(c);
      int bi, wl;
      singular = !warp_pivot(c, lane < nb && pos >= i, pos, bi, wl) || singular;
      pinv.x = __shfl_sync(0xffffffffu, pinv.x, wl);
      pinv.y = __shfl_sync(0xffffffffu, pinv.y, wl);
      // the row that was at position i takes the pivot's old position
      if (lane == wl) {
        pos = i;
      } else if (pos == i) {
        pos = bi;
      }
      const bool elim = lane < nb && pos > i;
      const cplx l = mul_xx(c, pinv);
      // columns in two halves; within a live half all are computed (and the
      // finished ones left alone), so that their shuffles and products overlap
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        if (wib + 4 * (4 * h + 3) >= i) {
          cplx u[4];
#pragma unroll
          for (int t = 0; t < 4; ++t) {
            u[t].x = __shfl_sync(0xffffffffu, x[4 * h + t].x, wl);
            u[t].y = __shfl_sync(0xffffffffu, x[4 * h + t].y, wl);
          }
#pragma unroll
          for (int t = 0; t < 4; ++t) {
            const int k = wib + 4 * (4 * h + t);
            cplx v = csub(x[4 * h + t], mul_xy(l, u[t]));
            v = (k == i) ? l : v;
            if (elim && k >= i) {
              x[4 * h + t] = v;
            }
            if (k == i + 1) {
              colbuf[k & 1][lane] = x[4 * h + t];
            }
          }
        }
      }
      __syncthreads();
    }
    // factors in position order
    if (lane < nb) {
#pragma unroll
      for (int t = 0; t < NBM / 4; ++t) {
        const int k = wib + 4 * t;
        if (k < nb) {
          Qm[pos * LD + k] = x[t];
          if (k == pos) {
            uinv[k] = cinv_lu(x[t]);
          }
        }
      }
      if (wib == 0) {
        at[pos] = lane;
      }
    }
    if (tid == 0 && singular) {
      atomicOr(&A.status[sl.grain], TMX_ST_SINGULAR);
    }
    __syncthreads();
    if (A.lu) {
      // factors and the column gather index, for the tangent solves
      cplx *Ls = A.lu + item.scratch;
      for (int u = tid; u < nb * nb; u += 128) {
        Ls[u] = Qm[(u / nb) * LD + (u % nb)];
      }
      int *ps = reinterpret_cast<int *>(Ls + (int64_t)nb * nb);
      if (tid < nb) {
        ps[tid] = pos; // (warp 0: lane = row)
      }
    }
    // ------------------------------------------ solve T_c Q_c = -RgQ_c
    // four lanes per row: row a, columns c + 4 t in y[t]
    const int a = tid >> 2, c = tid & 3;
    const bool act = a < nb;
    cplx y[NBM / 4];
#pragma unroll
    for (int t = 0; t < NBM / 4; ++t) {
      const int k = c + 4 * t;
      const cplx v = (act && k < nb) ? Rm[a * LD + k] : mkc(0., 0.);
      y[t] = mkc(-v.x, -v.y);
    }
    // Z U = X (forward over columns)
#pragma unroll
    for (int tj = 0; tj < NBM / 4; ++tj) {
      if (tj * 4 < nb) {
        for (int cj = 0; cj < 4; ++cj) {
          const int j = tj * 4 + cj;
          if (j >= nb) {
            break;
          }
          if (c == cj) {
            // (column 0: see mul_yx)
            y[tj] = (j == 0) ? mul_yx(y[tj], uinv[j]) : mul_xy(y[tj], uinv[j]);
          }
          cplx yj;
          yj.x = __shfl_sync(0xffffffffu, y[tj].x, cj, 4);
          yj.y = __shfl_sync(0xffffffffu, y[tj].y, cj, 4);
#pragma unroll
          for (int t = tj; t < NBM / 4; ++t) {
            const int k = c + 4 * t;
            if (k > j && k < nb) {
              y[t] = csub(y[t], mul_xy(yj, Qm[j * LD + k]));
            }
          }
        }
      }
    }
    // Y L = Z (backward over columns, L unit lower)
#pragma unroll
    for (int tj = NBM / 4 - 1; tj >= 0; --tj) {
      if (tj * 4 < nb) {
        for (int cj = min(4, nb - tj * 4) - 1; cj >= 0; --cj) {
          const int j = tj * 4 + cj;
          cplx yj;
          yj.x = __shfl_sync(0xffffffffu, y[tj].x, cj, 4);
          yj.y = __shfl_sync(0xffffffffu, y[tj].y, cj, 4);
#pragma unroll
          for (int t = 0; t <= tj; ++t) {
            const int k = c + 4 * t;
            if (k < j) {
              y[t] = csub(y[t], mul_xy(yj, Qm[j * LD + k]));
            }
          }
        }
      }
    }
    // write out: T_c[a][at[k]] = Y[a][k]
    if (act) {
      int ia, na;
      member(D, a, ia, na);
      if (sl.tout < 0) {
#pragma unroll
        for (int t = 0; t < NBM / 4; ++t) {
          const int k = c + 4 * t;
          if (k < nb && at[k] == a) {
            A.diag[sl.diag + ia * N + (na - 1)] = y[t];
          }
        }
      } else {
        cplx *Tr = A.tout + sl.tout + block_offset(N, m) +
                   (int64_t)(ia * D.nbb + (na - D.nmin)) * (2 * D.nbb);
#pragma unroll
        for (int t = 0; t < NBM / 4; ++t) {
          const int k = c + 4 * t;
          if (k < nb) {
            int ib, nbn;
            member(D, at[k], ib, nbn);
            Tr[ib * D.nbb + (nbn - D.nmin)] = y[t];
          }
        }
      }
    }
    __syncthreads(); // shared memory is reused by the next item
  }
}

static void launch_cta32(const TmxBlockArgs &a, cudaStream_t stream) {
  const size_t smem = (size_t)Cta32::ELEMS * sizeof(cplx);
  cudaFuncSetAttribute(k_blocks_cta32, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       (int)smem);
  // one item per CTA (see launch_warp_variant)
  const int blocks = (a.max_ctas > 0) ? std::min(std::max(1, a.nitems), a.max_ctas)
                                       : std::max(1, a.nitems);
  k_blocks_cta32<<<blocks, 128, smem, stream>>>(a);
}

// -------------------------------------- assembly, factors and solves apart --
//
// Classes of more than 32 members: one item is too much for a CTA's registers
// and too little, in its factorisation, for a whole SM's FP64 pipe, and the
// large orders come a few grains at a time. So the assembly of an item is
// split over CTAs of 32 rows x 32 columns (k_assemble, Q and RgQ to the item's
// scratch), one CTA per item factors Q (k_factor), and the solves are split by
// rows again (k_solve).
// Measured (B200), one CTA per item for everything -> the three kernels: 1154
// items of 33..50 members, 66..100 nodes: 1.41 -> 0.50 + 0.13 + 0.16 ms; 1960
// items of 65..99 members, 198 nodes: 15.4 -> 5.96 + 1.10 + 1.59 ms; the m = 0
// classes of nine grains at orders 129..199: 1.42 -> 0.32 ms per order.
// k_assemble is bound by the issue of its build phase (32 x 64 tiles with two
// CTAs per SM took 0.53 and 6.9 ms; three chunks of table rows in flight
// instead of one 0.56 and 7.1), k_solve by the FP64 pipe and the chain of its
// columns.

#define TMX_ASM_ROWS 32
#define TMX_ASM_COLS 32
#define TMX_ASM_WG 8 // quadrature nodes per chunk

// row tiles of an item of at most max_nb members: each holds rows of one
// group only (classes of m >= 1 have groups of at most (nb + 1) / 2 rows)
__host__ __device__ constexpr int asm_row_tiles(int max_nb) {
  return 2 * (((max_nb + 1) / 2 + TMX_ASM_ROWS - 1) / TMX_ASM_ROWS);
}
__host__ __device__ constexpr int asm_col_tiles(int max_nb) {
  return (max_nb + TMX_ASM_COLS - 1) / TMX_ASM_COLS;
}

// LEAN as for a_side_row: the factors a_n applied to the finished entries.
//
// Eight warps share the 8 x 8 tiles of the CTA's 32 x 32 entries (whatever is
// left of them at the edges) evenly, each tile four DMMA accumulators: (j, y) x
// (re, im). The K dimension is (node, term): four terms of a node for m >= 1,
// two for m = 0 (mu = 0 removes terms 0 and 2), in ascending order; a DMMA
// rounds as the four fused multiply-adds in that order. Thread t builds row
// and column t % 32 of node t / 32 of a chunk;
// the table rows of the next chunk are copied (cp.async) meanwhile. F and W
// rows are padded by two entries, so that the four terms and two members that
// eight lanes read fall into distinct banks.
template <bool LEAN>
__global__ void __launch_bounds__(256, 3) k_assemble(TmxBlockArgs A, int rtiles, int ctiles) {
  constexpr int NR = TMX_ASM_ROWS, NC = TMX_ASM_COLS, WG = TMX_ASM_WG;
  constexpr int LDF = NR + 2, LDW = NC + 2;
  constexpr int NP = (NR + NC) * 3; // 16-byte pieces of a node: 3 per member
  constexpr int NTILE = NR * NC / 64 / 8; // tiles per warp
  static_assert(WG * NC == 256 && WG * NR <= 256 && NP <= 256, "thread layout");
  extern __shared__ __align__(16) unsigned char asm_sm[];
  cplx *Fs = reinterpret_cast<cplx *>(asm_sm);                 // [4 WG][LDF]
  cplx *Ws = Fs + 4 * WG * LDF;                                // [4 WG][LDW]
  double *stg = reinterpret_cast<double *>(Ws + 4 * WG * LDW); // [WG][NP] pieces
  double *stgS = stg + WG * NP * 2;                            // [WG] node scalars
  __shared__ double an_s[NR + NC]; // a_n of the row and column members
  const int tid = threadIdx.x;
  const int lane = tid & 31;
  const int warp = tid >> 5;
  const int q = lane & 3;
  const int rr = lane >> 2;
  const int tiles = rtiles * ctiles;
  const int ilo = A.range ? A.range[0] : 0;
  const int ihi = A.range ? min(A.range[1], A.nitems) : A.nitems;
  for (int64_t u0 = (int64_t)ilo * tiles + blockIdx.x; u0 < (int64_t)ihi * tiles;
       u0 += gridDim.x) {
    const TmxItem item = A.items[u0 / tiles];
    const int tile = (int)(u0 % tiles);
    const TmxSlot sl = A.slots[item.slot];
    const int N = sl.nmax;
    const int ng = sl.ngauss;
    const int m = item.m;
    const ClassDesc D = describe<1>(N, m, item.cls);
    const int nb = D.nb;
    // rows [r0, r0 + nr) of group rg, columns [c0, c0 + nc)
    const int n0 = (D.R0 + NR - 1) / NR;
    const int rt = tile / ctiles;
    const int rg = (rt < n0) ? 0 : 1;
    const int r0 = (rg == 0) ? rt * NR : D.R0 + (rt - n0) * NR;
    const int nr = min(NR, ((rg == 0) ? D.R0 : nb) - r0);
    const int c0 = (tile % ctiles) * NC;
    const int nc = min(NC, nb - c0);
    if (nb > A.max_nb || nr <= 0 || nc <= 0) {
      continue; // (k_factor flags classes above the launch's size)
    }
    const TmxGrain Gr = A.grains[sl.grain];
    const double *T = A.tab + sl.tab;
    const double *S = A.nsc + sl.nsc;
    const double *Wg = A.wig + A.wig_off[sl.wig_n] + (int64_t)m * ng * N * 2;
    const double k2 = Gr.k * Gr.k;
    const cplx k2mr = mkc(Gr.mr * k2, Gr.mi * k2);
    const int nt = (m == 0) ? 2 : 4; // terms per node
    // this thread's piece: of row member r0 + tid / 3 (tid < 3 NR) or column
    // member c0 + tid / 3 - NR, a half of its Bessel row or its Wigner pair
    const int pm = tid / 3, piece = tid - 3 * pm;
    const bool prow = pm < NR;
    const bool have = tid < NP && (prow ? pm < nr : pm - NR < nc);
    int pi, pn;
    member(D, prow ? r0 + pm : c0 + pm - NR, pi, pn);
    pn = have ? pn : 1;
    const double *src = (piece < 2)
                            ? T + (int64_t)(pn - 1) * TMX_NQ + (prow ? 0 : 4) + 2 * piece
                            : Wg + (int64_t)(pn - 1) * 2;
    const int stride = (piece < 2) ? N * TMX_NQ : 2 * N;
    const auto issue = [&](int g0) {
      if (have) {
        const double *sp = src + (int64_t)g0 * stride;
#pragma unroll
        for (int gl = 0; gl < WG; ++gl) {
          if (g0 + gl < ng) {
            cp16(stg + (gl * NP + tid) * 2, sp);
          }
          sp += stride;
        }
      }
      if (tid < WG * (TMX_NS / 2) && g0 + tid / (TMX_NS / 2) < ng) {
        cp16(stgS + 2 * tid, S + (int64_t)g0 * TMX_NS + 2 * tid);
      }
      cp_commit();
    };
    issue(0);
    // this thread's row and column of a chunk (padding up to whole 8 x 8 tiles
    // is built as zeros; it is contracted but not written out)
    const int fg = tid / NR, fm = tid % NR;
    const int wg = tid / NC, wm = tid % NC;
    const bool frow = tid < WG * NR && (fm & ~7) < nr;
    const bool wcol = (wm & ~7) < nc;
    int fi, fn, wi, wn;
    member(D, r0 + fm, fi, fn);
    member(D, c0 + wm, wi, wn);
    if (tid < NR + NC && (tid < NR ? tid < nr : tid - NR < nc)) {
      int ia, n;
      member(D, tid < NR ? r0 + tid : c0 + tid - NR, ia, n);
      an_s[tid] = a_n(n);
    }
    // this warp's tiles: fo, wo their first entries in F and W
    const int nct = (nc + 7) >> 3;
    const int ntl = ((nr + 7) >> 3) * nct;
    int fo[NTILE], wo[NTILE];
    double acc[NTILE][4][2];
#pragma unroll
    for (int i = 0; i < NTILE; ++i) {
      const int t = warp + 8 * i;
      fo[i] = q * LDF + (t / nct) * 8 + rr;
      wo[i] = q * LDW + (t % nct) * 8 + rr;
#pragma unroll
      for (int p = 0; p < 4; ++p) {
        acc[i][p][0] = acc[i][p][1] = 0.;
      }
    }
    for (int g0 = 0; g0 < ng; g0 += WG) {
      cp_wait_all();
      __syncthreads(); // the chunk's rows are there; F and W are free
      if (frow) {
        cplx v[4] = {mkc(0., 0.), mkc(0., 0.), mkc(0., 0.), mkc(0., 0.)};
        if (fm < nr && g0 + fg < ng) {
          const double *r = stg + (fg * NP + 3 * fm) * 2;
          const double2 x = *reinterpret_cast<const double2 *>(r);
          const double2 y = *reinterpret_cast<const double2 *>(r + 2);
          const double2 w = *reinterpret_cast<const double2 *>(r + 4);
          a_side_row<LEAN>(x.x, x.y, y.x, y.y, w.x, w.y, stgS + fg * TMX_NS, fn, v, 1, m,
                           LEAN ? 1. : an_s[fm]);
        }
        cplx *o = Fs + fg * nt * LDF + fm;
        if (m == 0) {
          o[0] = v[1];
          o[LDF] = v[3];
        } else {
          o[0] = v[0];
          o[LDF] = v[1];
          o[2 * LDF] = v[2];
          o[3 * LDF] = v[3];
        }
      }
      if (wcol) {
        cplx v[4] = {mkc(0., 0.), mkc(0., 0.), mkc(0., 0.), mkc(0., 0.)};
        if (wm < nc && g0 + wg < ng) {
          const double *r = stg + (wg * NP + 3 * (NR + wm)) * 2;
          const double2 x = *reinterpret_cast<const double2 *>(r);
          const double2 y = *reinterpret_cast<const double2 *>(r + 2);
          const double2 w = *reinterpret_cast<const double2 *>(r + 4);
          const BSide B = b_side_node<LEAN>(wn, m, x, y, w.x, w.y, stgS + wg * TMX_NS,
                                            LEAN ? 1. : an_s[NR + wm]);
          b_side_terms<LEAN>(B, (rg == 0) ? D.iA : D.iB, wi, m, k2, k2mr, v, 1);
        }
        cplx *o = Ws + wg * nt * LDW + wm;
        if (m == 0) {
          o[0] = v[1];
          o[LDW] = v[3];
        } else {
          o[0] = v[0];
          o[LDW] = v[1];
          o[2 * LDW] = v[2];
          o[3 * LDW] = v[3];
        }
      }
      __syncthreads();
      if (g0 + WG < ng) {
        issue(g0 + WG);
      }
      const int kmax = min(WG, ng - g0) * nt;
      for (int k0 = 0; k0 < kmax; k0 += 4) {
#pragma unroll
        for (int i = 0; i < NTILE; ++i) {
          if (warp + 8 * i < ntl) {
            const cplx f = Fs[fo[i] + k0 * LDF];
            const cplx w = Ws[wo[i] + k0 * LDW];
            dmma(acc[i][0][0], acc[i][0][1], f.x, w.x); // jr
            dmma(acc[i][1][0], acc[i][1][1], f.x, w.y); // ji
            dmma(acc[i][2][0], acc[i][2][1], f.y, w.x); // yr
            dmma(acc[i][3][0], acc[i][3][1], f.y, w.y); // yi
          }
        }
      }
    }
    // Q = G^j + i G^y, RgQ = G^j
    cplx *Qs = A.scratch + item.scratch;
    cplx *Rs = Qs + (int64_t)nb * nb;
#pragma unroll
    for (int i = 0; i < NTILE; ++i) {
      const int t = warp + 8 * i;
      const int row = (t / nct) * 8 + rr;
      if (t < ntl && row < nr) {
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int cl = (t % nct) * 8 + 2 * q + e;
          if (cl < nc) {
            const double jr = acc[i][0][e], ji = acc[i][1][e];
            const double yr = acc[i][2][e], yi = acc[i][3][e];
            const double sc = LEAN ? an_s[row] * an_s[NR + cl] : 1.;
            const int64_t o = (int64_t)(r0 + row) * nb + c0 + cl;
            Qs[o] = mkc((jr - yi) * sc, (ji + yr) * sc);
            Rs[o] = mkc(jr * sc, ji * sc);
          }
        }
      }
    }
    __syncthreads(); // stage and chunk buffers are reused by the next tile
  }
}

// Pivot of one column over the lanes' candidates c[a] (bit a of live) at
// positions pos[a], rows r[a]: the first position with the largest |c| (|c|^2
// decides unless others come within rounding, see warp_pivot). Gives the row p,
// its position bi, 1 / c and d of the row; returns whether the pivot is zero.
template <int NP>
__device__ __forceinline__ bool lane_pivot(const cplx (&c)[NP], const cplx (&d)[NP],
                                           const int (&pos)[NP], const int (&r)[NP],
                                           unsigned live, int &p, int &bi, cplx &pinv,
                                           cplx &dp) {
  const unsigned long long top = 1ull << 63;
  double t[NP], best = 0.;
  int lp = 0x7fffffff, lr = 0, wl;
  cplx lc = mkc(0., 0.), ld = lc;
  const auto pick = [&]() { // largest t of this lane, first position on ties
    best = 0.;
    lp = 0x7fffffff;
#pragma unroll
    for (int a = 0; a < NP; ++a) {
      t[a] = (t[a] >= 0.) ? t[a] : 0.; // (NaN is no candidate)
      if ((live >> a & 1u) && (lp == 0x7fffffff || t[a] > best ||
                               (t[a] == best && pos[a] < lp))) {
        best = t[a];
        lp = pos[a];
        lr = r[a];
        lc = c[a];
        ld = d[a];
      }
    }
  };
  bool zero = false;
#pragma unroll
  for (int a = 0; a < NP; ++a) {
    t[a] = fma(c[a].x, c[a].x, c[a].y * c[a].y);
  }
  pick();
  pinv = cinv_lu(lc);
  warp_argmax(live ? (unsigned long long)__double_as_longlong(best) | top : 0ull, lp, bi,
              wl);
  best = __shfl_sync(0xffffffffu, best, wl);
  unsigned close = 0;
#pragma unroll
  for (int a = 0; a < NP; ++a) {
    close += ((live >> a & 1u) && t[a] >= best * (1. - 0x1p-40)) ? 1u : 0u;
  }
  if (__reduce_add_sync(0xffffffffu, close) != 1u ||
      !(best > 0x1p-900 && best < 0x1p900)) {
#pragma unroll
    for (int a = 0; a < NP; ++a) {
      t[a] = cabs_dev(c[a]);
    }
    pick();
    pinv = cinv_lu(lc);
    warp_argmax(live ? (unsigned long long)__double_as_longlong(best) | top : 0ull, lp, bi,
                wl);
    zero = !(__shfl_sync(0xffffffffu, best, wl) > 0.);
  }
  p = __shfl_sync(0xffffffffu, lr, wl);
  pinv.x = __shfl_sync(0xffffffffu, pinv.x, wl);
  pinv.y = __shfl_sync(0xffffffffu, pinv.y, wl);
  dp.x = __shfl_sync(0xffffffffu, ld.x, wl);
  dp.y = __shfl_sync(0xffffffffu, ld.y, wl);
  return zero;
}

// LU of Q_c, one item per CTA, in shared memory (in the scratch itself for
// classes whose factors exceed it).
//
// Rows stay in place; at[s] is the row at position s (the pivot of step i is
// the first position with the largest |Q_ri|, as in Matrix::plu_inverse), so
// the rows still to be eliminated are those at positions above i. Steps go in
// pairs, with one barrier per pair, and warp 0 runs a pair ahead: while the
// other UW warps apply steps i and i + 1 to the columns from i + 4 on (one load
// and store per entry for both, the updates in the order of the steps), it
// updates columns i + 2 and i + 3, finds their pivots and writes their l. The
// second pivot row of a pair has not had the first step's update then: every
// reader makes it, and one warp stores it in the phase after. Warp 0 applies
// the exchanges of positions to at[] while the others still read it, so they
// take the rows at the exchanged positions from the posted exchanges instead.
// The factors go back to the scratch with their rows in place, and the row at
// each position beside them.
// Bound by the latency of warp 0's columns and, while many rows are left, by
// the shared-memory traffic of the updates. All warps searching and inverting
// the pivot themselves -> warp 0 one column ahead -> a pair ahead: 1154 items of
// 33..50 members 0.227 -> 0.134 -> 0.126 ms, 1960 items of 65..99 1.99 -> 1.44
// -> 1.10 ms, the m = 0 classes of nine grains at orders 129..199 0.151 ->
// 0.117 -> 0.098 ms. Measured and not taken (one column ahead): update warps
// only beside, not on, warp 0's scheduler (0.194 and 1.88 ms); three CTAs per SM
// for up to 64 members (0.153 ms).
template <int NBM, int UW, int MINB>
__global__ void __launch_bounds__(32 + 32 * UW, MINB)
    k_factor(TmxBlockArgs A, size_t smem_bytes) {
  constexpr int NTH = 32 + 32 * UW;
  constexpr int CT = NTH / 16; // row groups of the copies
  constexpr int RT = 2 * UW;   // row groups of the updates
  constexpr int NA = (NBM + RT - 1) / RT; // rows per thread
  extern __shared__ __align__(16) unsigned char fsm[];
  __shared__ int at[NBM];                // row at a position
  // pivot rows of a pair of steps, their positions, the rows that gave way
  __shared__ int prow[2][2], pbi[2][2], pold[2][2];
  const int tid = threadIdx.x;
  const int lane = tid & 31;
  const int tc = tid & 15;
  const int tr = tid >> 4;
  const int ilo = A.range ? A.range[0] : 0;
  const int ihi = A.range ? min(A.range[1], A.nitems) : A.nitems;
  for (int it = ilo + blockIdx.x; it < ihi; it += gridDim.x) {
    const TmxItem item = A.items[it];
    const TmxSlot sl = A.slots[item.slot];
    const ClassDesc D = describe<1>(sl.nmax, item.m, item.cls);
    const int nb = D.nb;
    if (nb <= 0) {
      continue;
    }
    if (nb > NBM || nb > A.max_nb) {
      if (tid == 0) {
        atomicOr(&A.status[sl.grain], TMX_ST_TOO_LARGE);
      }
      continue;
    }
    cplx *Qs = A.scratch + item.scratch;
    const int lds = nb | 1;
    // (one body per address space: generic accesses to shared memory are slower)
    const auto factors = [&](auto ip) {
      constexpr bool inplace = decltype(ip)::value;
      const int lda = inplace ? nb : lds;
      cplx *Am;
      if constexpr (inplace) {
        Am = Qs;
      } else {
        Am = reinterpret_cast<cplx *>(fsm);
      }
      if (!inplace) {
        for (int r = tr; r < nb; r += CT) {
          for (int k = tc; k < nb; k += 16) {
            Am[r * lda + k] = Qs[(int64_t)r * nb + k];
          }
        }
      }
      for (int j = tid; j < nb; j += NTH) {
        at[j] = j;
      }
      __syncthreads();
      bool flag = false; // (warp 0) a pivot was zero
      // columns j and j + 1 by warp 0: NP positions per lane; p0, p1: pivot rows
      // of the pair before (columns j - 2 and j - 1)
      const auto panel = [&](auto np, int j, int p0, int p1) {
        constexpr int NP = decltype(np)::value;
        const bool two = j + 1 < nb;
        cplx v[NP], w[NP];
        int r[NP], pos[NP];
        unsigned live = 0;
        cplx u0 = mkc(0., 0.), u1 = u0, x0 = u0, x1 = u0;
        if (j > 0) {
          const cplx lp = Am[p1 * lda + j - 2];
          u0 = Am[p0 * lda + j];
          u1 = csub(Am[p1 * lda + j], mul_xy(lp, u0));
          if (two) {
            x0 = Am[p0 * lda + j + 1];
            x1 = csub(Am[p1 * lda + j + 1], mul_xy(lp, x0));
          }
        }
#pragma unroll
        for (int a = 0; a < NP; ++a) {
          pos[a] = j + lane + 32 * a;
          const bool in = pos[a] < nb;
          live |= in ? 1u << a : 0u;
          r[a] = in ? at[pos[a]] : -1;
          const cplx *row = Am + (in ? r[a] : 0) * lda;
          v[a] = row[j];
          w[a] = two ? row[j + 1] : mkc(0., 0.);
          if (j > 0) {
            const cplx l0 = row[j - 2], l1 = row[j - 1];
            v[a] = csub(csub(v[a], mul_xy(l0, u0)), mul_xy(l1, u1));
            w[a] = csub(csub(w[a], mul_xy(l0, x0)), mul_xy(l1, x1));
          }
        }
        const int o0 = __shfl_sync(0xffffffffu, r[0], 0);
        int q0, b0;
        cplx pinv, x;
        flag = lane_pivot<NP>(v, w, pos, r, live, q0, b0, pinv, x) || flag;
#pragma unroll
        for (int a = 0; a < NP; ++a) {
          if (r[a] == q0) {
            live &= ~(1u << a);
          } else {
            v[a] = mul_xx(v[a], pinv);
            w[a] = csub(w[a], mul_xy(v[a], x));
          }
          if (r[a] >= 0) {
            Am[r[a] * lda + j] = v[a];
          }
          // the row that was at position j takes the pivot's old position
          pos[a] = (r[a] == o0) ? b0 : pos[a];
        }
        int q1 = -1, b1 = -1;
        if (two) {
          flag = lane_pivot<NP>(w, v, pos, r, live, q1, b1, pinv, x) || flag;
#pragma unroll
          for (int a = 0; a < NP; ++a) {
            if (r[a] >= 0) {
              Am[r[a] * lda + j + 1] =
                  (r[a] == q0 || r[a] == q1) ? w[a] : mul_xx(w[a], pinv);
            }
          }
        }
        if (lane == 0) {
          const int k = (j >> 1) & 1;
          prow[k][0] = q0;
          pbi[k][0] = b0;
          pold[k][0] = o0;
          prow[k][1] = q1;
          pbi[k][1] = b1;
          pold[k][1] = two ? ((b0 == j + 1) ? o0 : at[j + 1]) : -1;
        }
      };
      const auto columns = [&](int j, int p0, int p1) {
        if (nb - j <= 32) {
          panel(std::integral_constant<int, 1>{}, j, p0, p1);
        } else if (NBM <= 64 || nb - j <= 64) {
          panel(std::integral_constant<int, 2>{}, j, p0, p1);
        } else {
          panel(std::integral_constant<int, NBM / 32>{}, j, p0, p1);
        }
      };
      if (tid < 32) {
        columns(0, 0, 0);
      }
      __syncthreads();
      int d0 = 0, d1 = -1; // pivot rows of the pair before
      for (int i = 0; i < nb; i += 2) {
        const int k2 = (i >> 1) & 1;
        const int p0 = prow[k2][0], bi0 = pbi[k2][0], o0 = pold[k2][0];
        const int p1 = prow[k2][1], bi1 = pbi[k2][1], o1 = pold[k2][1];
        if (tid < 32) {
          if (lane == 0) {
            at[bi0] = o0;
            at[i] = p0;
            if (p1 >= 0) {
              at[bi1] = o1;
              at[i + 1] = p1;
            }
          }
          __syncwarp();
          if (i + 2 < nb) {
            columns(i + 2, p0, p1);
          }
        } else {
          if (d1 >= 0 && tr < 4) {
            // the second pivot row of the pair before, which the others read
            // without its first update until now
            const cplx lp = Am[d1 * lda + i - 2];
            for (int k = i + lane; k < nb; k += 32) {
              Am[d1 * lda + k] = csub(Am[d1 * lda + k], mul_xy(lp, Am[d0 * lda + k]));
            }
          }
          const int s0 = i + 2 + tr - 2;
          if (s0 < nb) {
            const cplx *pr0 = Am + p0 * lda, *pr1 = Am + p1 * lda;
            const cplx lp = pr1[i];
            cplx l0[NA], l1[NA], *row[NA];
#pragma unroll
            for (int a = 0; a < NA; ++a) {
              const int s = s0 + RT * a;
              row[a] = Am;
              l0[a] = l1[a] = mkc(0., 0.);
              if (s < nb) {
                row[a] = Am + ((s == bi1) ? o1 : (s == bi0) ? o0 : at[s]) * lda;
                l0[a] = row[a][i];
                l1[a] = row[a][i + 1];
              }
            }
            for (int k = i + 4 + tc; k < nb; k += 16) {
              const cplx u0 = pr0[k];
              const cplx u1 = csub(pr1[k], mul_xy(lp, u0));
              cplx v[NA];
#pragma unroll
              for (int a = 0; a < NA; ++a) {
                if (s0 + RT * a < nb) {
                  v[a] = row[a][k];
                }
              }
#pragma unroll
              for (int a = 0; a < NA; ++a) {
                if (s0 + RT * a < nb) {
                  row[a][k] = csub(csub(v[a], mul_xy(l0[a], u0)), mul_xy(l1[a], u1));
                }
              }
            }
          }
          d0 = p0;
          d1 = p1;
        }
        __syncthreads();
      }
      if (tid == 0 && flag) {
        atomicOr(&A.status[sl.grain], TMX_ST_SINGULAR);
      }
      int *ps = reinterpret_cast<int *>(Qs + 2 * (int64_t)nb * nb);
      for (int j = tid; j < nb; j += NTH) {
        ps[j] = at[j];
      }
      if (!inplace) {
        for (int r = tr; r < nb; r += CT) {
          for (int k = tc; k < nb; k += 16) {
            Qs[(int64_t)r * nb + k] = Am[r * lda + k];
          }
        }
      }
      if (A.lu) {
        // factors (unit-lower L below, U on and above the diagonal) and the
        // column gather index, for the tangent solves
        cplx *Ls = A.lu + item.scratch;
        for (int r = tr; r < nb; r += CT) {
          const cplx *s = Am + at[r] * lda;
          for (int k = tc; k < nb; k += 16) {
            Ls[(int64_t)r * nb + k] = s[k];
          }
        }
        int *pl = reinterpret_cast<int *>(Ls + (int64_t)nb * nb);
        for (int j = tid; j < nb; j += NTH) {
          pl[at[j]] = j;
        }
      }
    };
    if (NBM > 64 && (size_t)nb * lds * sizeof(cplx) > smem_bytes) {
      factors(std::true_type{});
    } else {
      factors(std::false_type{});
    }
    __syncthreads(); // shared memory is reused by the next item
  }
}

// Solve T_c Q_c = -RgQ_c with k_factor's factors: CTA per NTH / C rows of an
// item, C lanes per row, the row in registers (column c + C t in x[t] of lane
// c, steps in blocks of C columns so that x is indexed statically), the
// factors copied to shared memory in position order (read in place for
// classes whose factors exceed it).
template <int NBM, int NTH, int C>
__global__ void __launch_bounds__(NTH, (NBM > 64) ? 1 : 2)
    k_solve(TmxBlockArgs A, int chunks, size_t smem_bytes) {
  constexpr int NT = NBM / C;
  constexpr int ROWS = NTH / C;
  extern __shared__ __align__(16) unsigned char fsm[];
  __shared__ cplx uinv[NBM];
  __shared__ int at[NBM];
  const int tid = threadIdx.x;
  const int c = tid % C;
  const int ilo = A.range ? A.range[0] : 0;
  const int ihi = A.range ? min(A.range[1], A.nitems) : A.nitems;
  for (int64_t u0 = (int64_t)ilo * chunks + blockIdx.x; u0 < (int64_t)ihi * chunks;
       u0 += gridDim.x) {
    const TmxItem item = A.items[u0 / chunks];
    const TmxSlot sl = A.slots[item.slot];
    const int N = sl.nmax;
    const int m = item.m;
    const ClassDesc D = describe<1>(N, m, item.cls);
    const int nb = D.nb;
    const int a0 = (int)(u0 % chunks) * ROWS;
    if (nb > NBM || nb > A.max_nb || a0 >= nb) {
      continue;
    }
    const cplx *Qs = A.scratch + item.scratch;
    const cplx *Rs = Qs + (int64_t)nb * nb;
    const int *ps = reinterpret_cast<const int *>(Rs + (int64_t)nb * nb);
    const int lds = nb | 1;
    const bool inplace = (size_t)nb * lds * sizeof(cplx) > smem_bytes;
    for (int j = tid; j < nb; j += NTH) {
      const int p = ps[j];
      at[j] = p;
      uinv[j] = cinv_lu(Qs[(int64_t)p * nb + j]);
    }
    __syncthreads();
    cplx *Fm = reinterpret_cast<cplx *>(fsm);
    if (!inplace) {
      for (int j = tid >> 5; j < nb; j += NTH / 32) {
        const cplx *s = Qs + (int64_t)at[j] * nb;
        for (int k = tid & 31; k < nb; k += 32) {
          cp16(Fm + j * lds + k, s + k);
        }
      }
      cp_commit();
    }
    const int a = a0 + tid / C;
    const bool act = a < nb;
    cplx x[NT];
#pragma unroll
    for (int t = 0; t < NT; ++t) {
      const int k = c + C * t;
      const cplx v = (act && k < nb) ? Rs[(int64_t)a * nb + k] : mkc(0., 0.);
      x[t] = mkc(-v.x, -v.y);
    }
    cp_wait_all();
    __syncthreads();
    // Above 64 members a body for shared memory alone beside the general one
    // (1.59 against 1.79 ms for 1960 items of 65..99 members); up to 64 the
    // loads that it hoists cost registers (0.18 against 0.16 ms for 1154 items).
    const auto solves = [&](auto ip) {
      constexpr bool SPLIT = decltype(ip)::value;
      // Z U = X (forward over columns)
  #pragma unroll
      for (int tj = 0; tj < NT; ++tj) {
        if (tj * C < nb) {
          for (int cj = 0; cj < C; ++cj) {
            const int j = tj * C + cj;
            if (j >= nb) {
              break;
            }
            if (c == cj) {
              // (column 0 of the classes up to 64: see mul_yx)
              x[tj] = (NBM <= 64 && j == 0) ? mul_yx(x[tj], uinv[j]) : mul_xy(x[tj], uinv[j]);
            }
            cplx xj;
            xj.x = __shfl_sync(0xffffffffu, x[tj].x, cj, C);
            xj.y = __shfl_sync(0xffffffffu, x[tj].y, cj, C);
            const cplx *ur;
            if constexpr (SPLIT) {
              ur = reinterpret_cast<const cplx *>(fsm) + j * lds;
            } else {
              ur = inplace ? Qs + (int64_t)at[j] * nb : Fm + j * lds;
            }
  #pragma unroll
            for (int t = tj; t < NT; ++t) {
              const int k = c + C * t;
              if (k > j && k < nb) {
                x[t] = csub(x[t], mul_xy(xj, ur[k]));
              }
            }
          }
        }
      }
      // Y L = Z (backward over columns, L unit lower)
  #pragma unroll
      for (int tj = NT - 1; tj >= 0; --tj) {
        if (tj * C < nb) {
          for (int cj = min(C, nb - tj * C) - 1; cj >= 0; --cj) {
            const int j = tj * C + cj;
            cplx xj;
            xj.x = __shfl_sync(0xffffffffu, x[tj].x, cj, C);
            xj.y = __shfl_sync(0xffffffffu, x[tj].y, cj, C);
            const cplx *lr;
            if constexpr (SPLIT) {
              lr = reinterpret_cast<const cplx *>(fsm) + j * lds;
            } else {
              lr = inplace ? Qs + (int64_t)at[j] * nb : Fm + j * lds;
            }
  #pragma unroll
            for (int t = 0; t <= tj; ++t) {
              const int k = c + C * t;
              if (k < j) {
                x[t] = csub(x[t], mul_xy(xj, lr[k]));
              }
            }
          }
        }
      }
    };
    if (NBM > 64 && !inplace) {
      solves(std::true_type{});
    } else {
      solves(std::false_type{});
    }
    // write out: T_c[a][at[k]] = Y[a][k]
    if (act) {
      int ia, na;
      member(D, a, ia, na);
      if (sl.tout < 0) {
#pragma unroll
        for (int t = 0; t < NT; ++t) {
          const int k = c + C * t;
          if (k < nb && at[k] == a) {
            A.diag[sl.diag + ia * N + (na - 1)] = x[t];
          }
        }
      } else {
        cplx *Tr = A.tout + sl.tout + block_offset(N, m) +
                   (int64_t)(ia * D.nbb + (na - D.nmin)) * (2 * D.nbb);
#pragma unroll
        for (int t = 0; t < NT; ++t) {
          const int k = c + C * t;
          if (k < nb) {
            int ib, nbn;
            member(D, at[k], ib, nbn);
            Tr[ib * D.nbb + (nbn - D.nmin)] = x[t];
          }
        }
      }
    }
    __syncthreads(); // shared memory is reused by the next chunk
  }
}

// dynamic shared memory a CTA may use for the factors (227 KB per block, less
// the static arrays)
#define TMX_FACTOR_SMEM_MAX (221u * 1024u)

template <bool LEAN, int NBM, int UW, int MINB, int NTHS, int C>
static void launch_apart(const TmxBlockArgs &a, cudaStream_t stream) {
  const int max_nb = std::max(1, std::min(a.max_nb, NBM));
  const int rt = asm_row_tiles(max_nb), ct = asm_col_tiles(max_nb);
  const int chunks = (max_nb + NTHS / C - 1) / (NTHS / C);
  // one tile, item or row chunk per CTA (see launch_warp_variant)
  const auto ctas = [&](int per_item) {
    const int64_t n = (int64_t)std::max(1, a.nitems) * per_item;
    return (unsigned)((a.max_ctas > 0) ? std::min<int64_t>(n, a.max_ctas) : n);
  };
  constexpr size_t asm_smem =
      4 * TMX_ASM_WG * (TMX_ASM_ROWS + TMX_ASM_COLS + 4) * sizeof(cplx) +
      TMX_ASM_WG * ((TMX_ASM_ROWS + TMX_ASM_COLS) * 6 + TMX_NS) * sizeof(double);
  cudaFuncSetAttribute(k_assemble<LEAN>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       (int)asm_smem);
  k_assemble<LEAN><<<ctas(rt * ct), 256, asm_smem, stream>>>(a, rt, ct);
  // factors in shared memory up to 118 members, above that in the scratch
  const size_t smem = std::min<size_t>((size_t)max_nb * (max_nb | 1) * sizeof(cplx),
                                       TMX_FACTOR_SMEM_MAX);
  // (the limit, not this launch's size: another thread may set it in between)
  cudaFuncSetAttribute(k_factor<NBM, UW, MINB>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       (int)TMX_FACTOR_SMEM_MAX);
  cudaFuncSetAttribute(k_solve<NBM, NTHS, C>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       (int)TMX_FACTOR_SMEM_MAX);
  k_factor<NBM, UW, MINB><<<ctas(1), 32 + 32 * UW, smem, stream>>>(a, smem);
  k_solve<NBM, NTHS, C><<<ctas(chunks), NTHS, smem, stream>>>(a, chunks, smem);
}

int tmx_block_family_capacity(int family) {
  switch (family) {
  case TMX_BLOCKS_WARP_DFMA:
    return 8;
  case TMX_BLOCKS_WARP_DMMA:
    return 16;
  case TMX_BLOCKS_CTA32:
    return 32;
  case TMX_BLOCKS_CTA64:
    return 64;
  case TMX_BLOCKS_CTA:
    return TMX_MAX_NB;
  default:
    return 0;
  }
}

// The family given in a.family (set by the host's dispatch table), else the
// smallest one whose capacity covers a.max_nb. A family whose capacity is
// below an item's class size flags that grain TMX_ST_TOO_LARGE.
int tmx_launch_blocks(const TmxBlockArgs &a, cudaStream_t stream) {
  if (a.nitems <= 0) {
    return 0;
  }
  int f = a.family;
  if (f < 0 || f >= TMX_BLOCK_FAMILIES) {
    f = (a.max_nb <= 8)    ? TMX_BLOCKS_WARP_DFMA
        : (a.max_nb <= 16) ? TMX_BLOCKS_WARP_DMMA
        : (a.max_nb <= 32) ? TMX_BLOCKS_CTA32
        : (a.max_nb <= 64) ? TMX_BLOCKS_CTA64
                           : TMX_BLOCKS_CTA;
  }
  switch (f) {
  case TMX_BLOCKS_WARP_DFMA:
    launch_warp_variant<1, 2, TMX_WARP_DFMA_MINB, false>(a, stream);
    return 1;
  case TMX_BLOCKS_WARP_DMMA:
    launch_warp_variant<1, 1, TMX_WARP_DMMA_MINB, true>(a, stream);
    return 1;
  case TMX_BLOCKS_CTA32:
    launch_cta32(a, stream);
    return 1;
  case TMX_BLOCKS_CTA64:
    launch_apart<true, 64, 8, 2, 512, 8>(a, stream);
    return 3;
  default:
    launch_apart<false, 128, 15, 1, 512, 16>(a, stream);
    return 3;
  }
}

// ----------------------------------------------------------- convergence --

// The m = 0 sums of every (active slot, order of the group), one thread each,
// in the reference's order (TMatrixResource.hpp:743-756); then one thread per
// slot applies the convergence test (:758-775) order by order until the order
// is final. Unconverged slots that have orders left go to the next list.
// One launch per group: with few grains left the kernels of the loop are
// shorter than their launches (eight orders of one grain: eight of 3 us -> one
// of 6 us). Bound by the latency of the diagonal's loads: CV_LOADS orders are
// read ahead of their additions.
#define CV_THREADS 128
#define CV_LOADS 8
__global__ void k_converge(const int32_t *__restrict__ active, int nactive,
                           const __grid_constant__ TmxChainGroup g, int lg,
                           const TmxSlot *__restrict__ slots,
                           const cplx *__restrict__ diag, TmxChainState *state,
                           double tolerance, int last_order,
                           int32_t *next_active, int32_t *next_count,
                           int32_t *done_list, int32_t *done_ord,
                           int32_t *done_pos, int32_t *done_count,
                           const int32_t *nact_dev, int base) {
  __shared__ double sq[CV_THREADS], se[CV_THREADS];
  // order s of the group and slot p: 2^lg threads per slot
  const int s = threadIdx.x & ((1 << lg) - 1);
  const int p = (blockIdx.x * CV_THREADS + threadIdx.x) >> lg;
  const bool have = p < nactive && (!nact_dev || base + p < *nact_dev);
  int gr = 0;
  TmxChainState st;
  if (have && s == 0) { // (read beside the sums)
    gr = active[p];
    st = state[gr];
  }
  if (have && s < g.n) {
    const TmxSlot sl = slots[g.base[s].slot + p];
    const cplx *dg = diag + sl.diag;
    const int N = g.order0 + s;
    double qs = 0., qe = 0.;
    for (int n0 = 1; n0 < N + 1; n0 += CV_LOADS) {
      cplx a[CV_LOADS], b[CV_LOADS];
#pragma unroll
      for (int i = 0; i < CV_LOADS; ++i) {
        const int n = min(n0 + i, N);
        a[i] = dg[n - 1];
        b[i] = dg[N + n - 1];
      }
#pragma unroll
      for (int i = 0; i < CV_LOADS; ++i) {
        if (n0 + i < N + 1) {
          const double dn1 = 2. * (n0 + i) + 1.;
          qs += dn1 * (cnorm2(a[i]) + cnorm2(b[i]));
          qe += dn1 * (a[i].x + b[i].x);
        }
      }
    }
    sq[threadIdx.x] = qs;
    se[threadIdx.x] = qe;
  }
  __syncthreads();
  if (!have || s != 0) {
    return;
  }
  bool stays = false;
  for (int t = 0; t < g.n; ++t) {
    const double qs = sq[threadIdx.x + t], qe = se[threadIdx.x + t];
    const int order = g.order0 + t;
    const double old_qs = st.qsca, old_qe = st.qext;
    st.qsca = qs;
    st.qext = qe;
    st.nmax = order;
    st.ngauss = g.glf * order;
    if (st.dqs_t == -2.) {
      st.dqs_t = -1.;
      st.dqe_t = -1.;
    } else {
      st.dqs_t = fabs((old_qs - qs) / qs);
      st.dqe_t = fabs((old_qe - qe) / qe);
    }
    if (st.dqs_t > 0.) {
      st.dqs = st.dqs_t;
      st.dqe = st.dqe_t;
      if (st.dqs_t <= tolerance && st.dqe_t <= tolerance) {
        st.converged = 1;
      }
    }
    const bool finite = isfinite(qs) && isfinite(qe);
    if (!finite) {
      st.status |= TMX_ST_NAN;
    }
    stays = !st.converged && finite && order < last_order;
    if (!st.converged && finite && !stays) {
      st.status |= TMX_ST_NOT_CONVERGED;
    }
    if (!stays) {
      break;
    }
  }
  state[gr] = st;
  if (stays) {
    const int q = atomicAdd(next_count, 1);
    next_active[q] = gr;
  } else {
    // the grain's order is final: its blocks may start
    const int q = atomicAdd(done_count, 1);
    done_list[q] = gr;
    done_ord[q] = st.nmax;
    done_pos[q] = p;
  }
}

void tmx_launch_converge(const int32_t *active, int nactive, const TmxChainGroup &g,
                         const TmxSlot *slots, const double2 *diag,
                         TmxChainState *state, double tolerance, int last_order,
                         int32_t *next_active, int32_t *next_count,
                         int32_t *done_list, int32_t *done_ord, int32_t *done_pos,
                         int32_t *done_count, const int32_t *nact_dev, int base,
                         cudaStream_t stream) {
  if (nactive <= 0) {
    return;
  }
  const int lg = g.n <= 1 ? 0 : g.n <= 2 ? 1 : g.n <= 4 ? 2 : 3;
  const int per = CV_THREADS >> lg;
  k_converge<<<(nactive + per - 1) / per, CV_THREADS, 0, stream>>>(
      active, nactive, g, lg, slots, diag, state, tolerance, last_order, next_active,
      next_count, done_list, done_ord, done_pos, done_count, nact_dev, base);
}

// ------------------------------------------------------------- kept tables --

// The node scalars and Bessel tables of a grain's final order are the ones
// its block round needs. Right after the convergence test of a group of
// orders (before the next group overwrites the order loop's table buffers),
// every grain that became final in the group -- done-list entries
// [*next, counters[1]) -- has its tables copied into the batch's arena at a
// reserved offset (in doubles, a multiple of 16), recorded per grain and per
// done-list entry; -1 where the arena is full (the round then recomputes
// them). One CTA per entry, grid-stride; the last CTA to finish moves *next
// to the end of the range. Part of the order loop's chain and bound by the
// latency of its loads (13 to 130 KB per entry): 512 threads with four 16-byte
// loads in flight each, the first ones beside the reservation. 4096 grains,
// 19 launches: 453 -> 184 us (128 threads, one load after the other: up to
// 42 us for the 115 KB of an order 30); the batch 5.85 -> 5.30 ms together
// with the loads of k_converge (203 -> 173 us).
#define KT_THREADS 512
#define KT_LOADS 4
__global__ void __launch_bounds__(KT_THREADS)
    k_keep_tables(const __grid_constant__ TmxKeepArgs K) {
  __shared__ long long s_off;
  __shared__ unsigned s_last;
  const int order0 = K.order0_dev ? *K.order0_dev : K.order0;
  const int begin = *K.next;
  const int end = K.counters[1];
  for (int q = begin + blockIdx.x; q < end; q += gridDim.x) {
    const int g = K.done_list[q];
    const int s = K.done_ord[q] - order0;
    const int p = K.done_pos[q];
    const TmxChainBase &b = K.order0_dev ? *K.base_dev : K.base[s];
    const int64_t tsz = b.tab_stride, nsz = b.nsc_stride;
    const int64_t tpad = (tsz + 15) & ~(int64_t)15;
    const int64_t want = tpad + ((nsz + 15) & ~(int64_t)15);
    if (threadIdx.x == 0) {
      const long long off =
          (long long)atomicAdd(K.used, (unsigned long long)want);
      s_off = (off + want <= K.cap) ? off : -1;
    }
    const double2 *ts = reinterpret_cast<const double2 *>(K.tab + b.tab + p * tsz);
    const double2 *ns = reinterpret_cast<const double2 *>(K.nsc + b.nsc + p * nsz);
    const int nt = (int)(tsz / 2), nn = nt + (int)(nsz / 2);
    double2 v[KT_LOADS];
    const auto load = [&](int u0) {
#pragma unroll
      for (int i = 0; i < KT_LOADS; ++i) {
        const int u = u0 + i * KT_THREADS;
        if (u < nn) {
          v[i] = u < nt ? ts[u] : ns[u - nt];
        }
      }
    };
    load(threadIdx.x); // (beside the reservation)
    __syncthreads();
    const long long off = s_off;
    if (off >= 0) {
      double2 *td = reinterpret_cast<double2 *>(K.arena + off);
      double2 *nd = reinterpret_cast<double2 *>(K.arena + off + tpad);
      for (int u0 = threadIdx.x; u0 < nn; u0 += KT_LOADS * KT_THREADS) {
        if (u0 != threadIdx.x) {
          load(u0);
        }
#pragma unroll
        for (int i = 0; i < KT_LOADS; ++i) {
          const int u = u0 + i * KT_THREADS;
          if (u < nn) {
            *(u < nt ? td + u : nd + (u - nt)) = v[i];
          }
        }
      }
    }
    if (threadIdx.x == 0) {
      K.keep_tab[g] = off;
      K.keep_q[q] = off;
    }
    __syncthreads();
  }
  // the last CTA moves the start of the next range
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    s_last = (atomicAdd(K.ticket, 1u) == gridDim.x - 1) ? 1u : 0u;
  }
  __syncthreads();
  if (s_last && threadIdx.x == 0) {
    *K.next = end;
    *K.ticket = 0u;
    __threadfence();
  }
}

void tmx_launch_keep_tables(const TmxKeepArgs &K, int max_entries,
                            cudaStream_t stream) {
  const int blocks = std::max(1, std::min(max_entries, 148 * 4));
  k_keep_tables<<<blocks, KT_THREADS, 0, stream>>>(K);
}

// ------------------------------------------------------------- Q sums ------

// TMatrixQTask::execute (TMatrixResource.hpp:1136-1210): full Qsca and Qext.
// The reference's quadruple loop over (n1, n2, m1, m2 = m1) visits every
// entry of every m block once, so Qsca = sum_m f_m ||T_m||_F^2 and
// Qext = sum_m f_m sum_n Re(T_m[(0,n),(0,n)] + T_m[(0,n),(1,n)] +
// T_m[(1,n),(0,n)] + T_m[(1,n),(1,n)]), f_0 = 1, f_m = 2.
//
// A grain's blocks are one contiguous range of T, so |T|^2 is summed over that
// range without regard to blocks (weight 1 up to the end of block 0, 2 after
// it), all loads of a thread independent; the diagonals are read on their own,
// a warp per block. Grains of more than 24 orders are shared by 4 or 16 CTAs
// (blockIdx.y): the last one to finish adds the partial sums in order, so the
// result depends on the grain alone. Bound by reading T: 28 grains of order 99
// (21 MB each) 1.99 -> 0.15 ms, 96 grains of orders 16..50 0.28 -> 0.038 ms
// against one CTA per grain that went block by block.
#define QS_THREADS 256
__host__ __device__ static inline int qsum_parts(int N) {
  return N <= 24 ? 1 : N <= 48 ? 4 : TMX_QSUM_PARTS;
}

__global__ void __launch_bounds__(QS_THREADS)
    k_qsums(const TmxSlot *__restrict__ slots, int ns, const cplx *__restrict__ T,
            double *q_out, double *part, unsigned *ticket,
            const int32_t *__restrict__ range) {
  __shared__ double red[2][QS_THREADS / 32];
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int slo = range ? range[0] : 0;
  const int shi = range ? min(range[1], ns) : ns;
  for (int s = slo + blockIdx.x; s < shi; s += gridDim.x) {
    const TmxSlot sl = slots[s];
    const int N = sl.nmax;
    const int np = qsum_parts(N);
    const int ip = blockIdx.y;
    if (ip >= np) {
      continue;
    }
    const cplx *Tg = T + sl.tout;
    double qs = 0., qe = 0.;
    if (N > 0) {
      const int64_t total = block_offset(N, N + 1);
      const int64_t first = 4 * (int64_t)N * N;
      const int64_t chunk = (total + np - 1) / np;
      const int64_t end = min(total, (ip + 1) * chunk);
#pragma unroll 4
      for (int64_t u = ip * chunk + threadIdx.x; u < end; u += QS_THREADS) {
        const cplx v = Tg[u];
        qs += (u < first) ? cnorm2(v) : 2. * cnorm2(v);
      }
      for (int m = ip * (QS_THREADS / 32) + warp; m <= N; m += np * (QS_THREADS / 32)) {
        const int nb = (m == 0) ? N : N + 1 - m;
        const int w = 2 * nb;
        const cplx *B = Tg + block_offset(N, m);
        double be = 0.;
        for (int r = lane; r < nb; r += 32) {
          const cplx *d = B + (int64_t)r * w + r;
          const cplx *e = d + (int64_t)nb * w;
          be += (d[0].x + d[nb].x) + (e[0].x + e[nb].x);
        }
        qe += (m > 0) ? 2. * be : be;
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      qs += __shfl_down_sync(0xffffffffu, qs, o);
      qe += __shfl_down_sync(0xffffffffu, qe, o);
    }
    if (lane == 0) {
      red[0][warp] = qs;
      red[1][warp] = qe;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      double a = 0., b = 0.;
      for (int i = 0; i < QS_THREADS / 32; ++i) {
        a += red[0][i];
        b += red[1][i];
      }
      if (np == 1) {
        q_out[2 * sl.grain] = a;
        q_out[2 * sl.grain + 1] = b;
      } else {
        volatile double *pg = part + (int64_t)sl.grain * 2 * TMX_QSUM_PARTS;
        pg[2 * ip] = a;
        pg[2 * ip + 1] = b;
        __threadfence();
        if (atomicAdd(&ticket[sl.grain], 1u) == (unsigned)(np - 1)) {
          __threadfence();
          a = b = 0.;
          for (int i = 0; i < np; ++i) {
            a += pg[2 * i];
            b += pg[2 * i + 1];
          }
          q_out[2 * sl.grain] = a;
          q_out[2 * sl.grain + 1] = b;
          ticket[sl.grain] = 0u; // ready for the grain's next batch
        }
      }
    }
    // red is reused by the next slot
    __syncthreads();
  }
}

size_t tmx_qsum_part_bytes(int64_t n) {
  return (size_t)n * (2 * TMX_QSUM_PARTS * sizeof(double) + sizeof(unsigned));
}

void tmx_launch_qsums(const TmxSlot *slots, int ns, const cplx *T, double *q_out,
                      double *part, int64_t n, int nmax, cudaStream_t stream,
                      const int32_t *range, int max_ctas) {
  if (ns <= 0) {
    return;
  }
  const int blocks = (max_ctas > 0) ? std::min(ns, max_ctas) : ns;
  unsigned *ticket = reinterpret_cast<unsigned *>(part + 2 * TMX_QSUM_PARTS * n);
  k_qsums<<<dim3(blocks, qsum_parts(nmax)), QS_THREADS, 0, stream>>>(
      slots, ns, T, q_out, part, ticket, range);
}

// ------------------------------------------------------------ chain prep --

// Slots and items of a group of orders (blockIdx.y): active position p gets the
// tables at p * strides and the four m = 0 classes as items 4p .. 4p + 3.
__global__ void k_chain_prep(const int32_t *__restrict__ active, int nactive,
                             const int32_t *__restrict__ nact_dev, int base,
                             const __grid_constant__ TmxChainGroup g, TmxSlot *slots,
                             TmxItem *items) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= nactive) {
    return;
  }
  const TmxChainBase &b = g.base[blockIdx.y];
  const int order = g.order0 + (int)blockIdx.y;
  // positions past the list's length on the device (the host launched for
  // an upper bound) get an empty slot: order 0 has no classes and no nodes,
  // so every kernel of the step skips it
  const bool valid = !nact_dev || base + p < *nact_dev;
  TmxSlot s;
  s.grain = valid ? active[p] : 0;
  s.nmax = valid ? order : 0;
  s.ngauss = valid ? g.glf * order : 0;
  s.wig_n = g.wig[blockIdx.y];
  s.tab = b.tab + p * b.tab_stride;
  s.nsc = b.nsc + p * b.nsc_stride;
  s.tout = -1;
  s.diag = b.diag + p * b.diag_stride;
  slots[b.slot + p] = s;
  for (int c = 0; c < 4; ++c) {
    TmxItem it;
    it.slot = b.slot + p;
    it.m = 0;
    it.cls = (int16_t)c;
    it.scratch = b.scr + (4 * (int64_t)p + c) * b.scr_stride;
    items[4 * (b.slot + p) + c] = it;
  }
}

void tmx_launch_chain_prep(const int32_t *active, int nactive,
                           const int32_t *nact_dev, int base,
                           const TmxChainGroup &g, TmxSlot *slots, TmxItem *items,
                           cudaStream_t stream) {
  if (nactive <= 0) {
    return;
  }
  k_chain_prep<<<dim3((nactive + 127) / 128, g.n), 128, 0, stream>>>(
      active, nactive, nact_dev, base, g, slots, items);
}

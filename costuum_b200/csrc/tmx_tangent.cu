// Tangent (forward-mode derivative) kernel of the T-matrix blocks.
//
// For p in {refractive index m (complex derivative), equal-volume radius
// R_V, axis ratio d} and every (grain, m, class) item:
//   dT_c = -(dRgQ_c + T_c dQ_c) Q_c^-1,
// differentiating T_c Q_c = -RgQ_c (the relation T = -RgQ Q^-1 of
// TMatrixResource.hpp:712-730, 1102-1119) and reusing the LU factors of Q_c
// saved by the forward block kernel. The entries of Q and RgQ are
// sum_g sum_t F_t W_t (see tmx_blocks.cu), so dQ = sum [dF W + F dW]: the
// same contraction with the node dimension doubled. All derivatives are
// algebraic in the forward tables; for a spherical Bessel function f of
// argument z and its derivative form df = [z f]'/z (SpecialFunctions.hpp:
// 106-240) the Bessel equation z^2 f'' + 2 z f' + (z^2 - n(n+1)) f = 0 gives
//   d f/dz = df - f/z,   d(df)/dz = n(n+1) f / z^2 - f - df / z.
// Arguments: z = k R_V r(theta), w = m z; dz/dR_V = z/R_V, dw/dm = z,
// dw/dR_V = w/R_V, dz/dd = z (dln r^2/dd)/2; the quadrature weights w r^2
// (and m w r^2 / sin) scale with r^2, so d/dd multiplies them by dln r^2/dd;
// r'/r also depends on d.
#include <algorithm>

#include "tmx_blocks_common.cuh"

extern __shared__ __align__(16) unsigned char tmx_tsmem[];

enum { P_M = 0, P_R = 1, P_D = 2 };

// Tangent chunk: per node 8 slots, slot t (t < 4) pairs F_t with dW_t and
// slot 4 + t pairs dF_t with W_t. For p = m the F side does not depend on
// the parameter and only slots 0..3 are used.
// Threads tid = 0..nth-1 of the caller share the work; rows are stored with
// stride L.NRp, columns with stride ncolp. an_tab[a] = a_n of member a.
__device__ void build_chunk_tangent(const ClassDesc &D, const AsmLayout &L,
                                    int ncolp, int N, int m, int ng, int g0,
                                    int param, double R,
                                    const double *__restrict__ T,
                                    const double *__restrict__ S,
                                    const double *__restrict__ Wg, double k2,
                                    cplx k2mr, cplx *Fs, cplx *Ws, int tid,
                                    int nth, const double *an_tab) {
  const int G = L.G;
  const int slots = 8;
  // ---- A side: F_t (slots 0..3) and dF_t (slots 4..7), (F^j, F^y) pairs
  for (int u = tid; u < G * L.NRp; u += nth) {
    const int gl = u / L.NRp;
    const int pr = u % L.NRp;
    const int g = g0 + gl;
    const int a = padded_member(D, pr);
    cplx f[4], df[4];
    for (int t = 0; t < 4; ++t) {
      f[t] = df[t] = mkc(0., 0.);
    }
    if (a >= 0 && g < ng) {
      int i, n;
      member(D, a, i, n);
      const double *tb = T + ((int64_t)g * N + (n - 1)) * TMX_NQ;
      const double *w = Wg + ((int64_t)g * N + (n - 1)) * 2;
      const double *s = S + (int64_t)g * TMX_NS;
      const double d = w[0], dd = w[1];
      const double an = an_tab[a];
      const double nn = n * (n + 1.);
      const double iz = s[TMX_NS_KRINV];
      const double drr = s[TMX_NS_DRR];
      // h = (j, y) parts handled together
      const double hj = tb[TMX_Q_J], hy = tb[TMX_Q_Y];
      const double dhj = tb[TMX_Q_DJ], dhy = tb[TMX_Q_DY];
      const double q = nn * drr * iz * d;
      f[0] = mkc(an * d * hj, an * d * hy);
      f[1] = mkc(an * dd * hj, an * dd * hy);
      f[2] = mkc(an * d * dhj, an * d * dhy);
      f[3] = mkc(an * (dd * dhj + q * hj), an * (dd * dhy + q * hy));
      if (param != P_M) {
        // d/dz of h, dh and h/z
        const double hpj = dhj - hj * iz, hpy = dhy - hy * iz;
        const double dhpj = nn * hj * iz * iz - hj - dhj * iz;
        const double dhpy = nn * hy * iz * iz - hy - dhy * iz;
        const double hzpj = dhj * iz - 2. * hj * iz * iz;
        const double hzpy = dhy * iz - 2. * hy * iz * iz;
        const double z = s[TMX_NS_KR];
        const double dz = (param == P_R) ? z / R : 0.5 * z * s[TMX_NS_DLNR2_DD];
        const double ddrr = (param == P_D) ? s[TMX_NS_DDRR_DD] : 0.;
        df[0] = mkc(an * d * hpj * dz, an * d * hpy * dz);
        df[1] = mkc(an * dd * hpj * dz, an * dd * hpy * dz);
        df[2] = mkc(an * d * dhpj * dz, an * d * dhpy * dz);
        df[3] = mkc(an * ((dd * dhpj + nn * drr * d * hzpj) * dz +
                          nn * ddrr * d * hj * iz),
                    an * ((dd * dhpy + nn * drr * d * hzpy) * dz +
                          nn * ddrr * d * hy * iz));
      }
    }
    cplx *fp = Fs + (int64_t)(slots * gl) * L.NRp + pr;
    for (int t = 0; t < 4; ++t) {
      fp[t * L.NRp] = f[t];
      fp[(4 + t) * L.NRp] = df[t];
    }
  }
  // ---- B side: dW_t (slots 0..3) and W_t (slots 4..7) for each row group
  for (int u = tid; u < G * ncolp; u += nth) {
    const int gl = u / ncolp;
    const int b = u % ncolp;
    const int g = g0 + gl;
    cplx W[2][4], dW[2][4];
    for (int rg = 0; rg < 2; ++rg) {
      for (int t = 0; t < 4; ++t) {
        W[rg][t] = dW[rg][t] = mkc(0., 0.);
      }
    }
    if (b < D.nb && g < ng) {
      int ib, n;
      member(D, b, ib, n);
      const double *tb = T + ((int64_t)g * N + (n - 1)) * TMX_NQ;
      const cplx jm = mkc(tb[TMX_Q_JM_RE], tb[TMX_Q_JM_IM]);
      const cplx djm = mkc(tb[TMX_Q_DJM_RE], tb[TMX_Q_DJM_IM]);
      const double *w = Wg + ((int64_t)g * N + (n - 1)) * 2;
      const double *s = S + (int64_t)g * TMX_NS;
      const double d = w[0], dd = w[1];
      const double an = an_tab[b];
      const double nn = n * (n + 1.);
      const cplx iw = mkc(s[TMX_NS_KRMRINV_RE], s[TMX_NS_KRMRINV_IM]);
      const double drr = s[TMX_NS_DRR];
      const cplx jw = cmul(jm, iw); // j / w
      const cplx Gv[4] = {
          cscale(djm, an * d),
          cscale(cadd(cscale(djm, dd), cscale(jw, drr * nn * d)), an),
          cscale(jm, an * d), cscale(jm, an * dd)};
      // d/dw of j, dj and j/w
      const cplx iw2 = cmul(iw, iw);
      const cplx jp = csub(djm, jw);
      const cplx djp = csub(csub(cscale(cmul(jm, iw2), nn), jm), cmul(djm, iw));
      const cplx jwp = csub(cmul(djm, iw), cscale(cmul(jm, iw2), 2.));
      // dw/dp
      const cplx wv = mkc(s[TMX_NS_KRMR_RE], s[TMX_NS_KRMR_IM]);
      cplx dw;
      if (param == P_M) {
        dw = mkc(s[TMX_NS_KR], 0.);
      } else if (param == P_R) {
        dw = cscale(wv, 1. / R);
      } else {
        dw = cscale(wv, 0.5 * s[TMX_NS_DLNR2_DD]);
      }
      const double ddrr = (param == P_D) ? s[TMX_NS_DDRR_DD] : 0.;
      const cplx dGv[4] = {
          cmul(cscale(djp, an * d), dw),
          cadd(cmul(cscale(cadd(cscale(djp, dd), cscale(jwp, drr * nn * d)), an), dw),
               cscale(jw, an * nn * d * ddrr)),
          cmul(cscale(jp, an * d), dw), cmul(cscale(jp, an * dd), dw)};
      const double wr2 = s[TMX_NS_W] * s[TMX_NS_R2];
      const double mu = (double)(m * m) * s[TMX_NS_SIN2INV];
      const double beta = s[TMX_NS_SININV] * m * wr2;
      // d(weight)/dp / weight: r^2 scales the weights when d changes
      const double lw = (param == P_D) ? s[TMX_NS_DLNR2_DD] : 0.;
      const cplx k2c = mkc(k2, 0.);
      const cplx dk2mr = (param == P_M) ? k2c : mkc(0., 0.);
      for (int rg = 0; rg < L.ngroups; ++rg) {
        const int ia = (rg == 0) ? D.iA : D.iB;
        if (ia == ib) {
          const cplx chi = (ia == 0) ? k2mr : k2c;
          const cplx clo = (ia == 0) ? mkc(-k2, 0.) : mkc(-k2mr.x, -k2mr.y);
          const cplx dchi = (ia == 0) ? dk2mr : mkc(0., 0.);
          const cplx dclo = (ia == 0) ? mkc(0., 0.) : mkc(-dk2mr.x, -dk2mr.y);
          const double wts[4] = {wr2 * mu, wr2, wr2 * mu, wr2};
          for (int t = 0; t < 4; ++t) {
            const cplx c = (t < 2) ? chi : clo;
            const cplx dc = (t < 2) ? dchi : dclo;
            W[rg][t] = cmul(c, cscale(Gv[t], wts[t]));
            // d(c w G) = dc w G + c (lw w) G + c w dG
            dW[rg][t] = cadd(cmul(dc, cscale(Gv[t], wts[t])),
                             cmul(c, cadd(cscale(Gv[t], wts[t] * lw),
                                          cscale(dGv[t], wts[t]))));
          }
        } else {
          const cplx c1 = (ia == 0) ? k2mr : k2c;
          const cplx c2 = (ia == 0) ? k2c : k2mr;
          const cplx dc1 = (ia == 0) ? dk2mr : mkc(0., 0.);
          const cplx dc2 = (ia == 0) ? mkc(0., 0.) : dk2mr;
          const int gi[4] = {3, 2, 1, 0};
          for (int t = 0; t < 4; ++t) {
            const cplx c = (t < 2) ? c1 : c2;
            const cplx dc = (t < 2) ? dc1 : dc2;
            const cplx ic = mkc(-c.y * beta, c.x * beta);    // i c beta
            const cplx idc = mkc(-dc.y * beta, dc.x * beta); // i dc beta
            const cplx Gt = Gv[gi[t]];
            W[rg][t] = cmul(ic, Gt);
            dW[rg][t] = cadd(cmul(idc, Gt),
                             cmul(ic, cadd(cscale(Gt, lw), dGv[gi[t]])));
          }
        }
      }
    }
    for (int rg = 0; rg < L.ngroups; ++rg) {
      cplx *wp = Ws + ((int64_t)rg * slots * G + slots * gl) * ncolp + b;
      for (int t = 0; t < 4; ++t) {
        wp[t * ncolp] = dW[rg][t];
        wp[(4 + t) * ncolp] = W[rg][t];
      }
    }
  }
}

// One block per (item, parameter): classes above 32 members.
template <int TR, int TC, int NT, int MINB>
__global__ void __launch_bounds__(NT, MINB)
    k_tangent(TmxTangentArgs A, size_t smem_bytes) {
  const int it = blockIdx.x;
  const int param = blockIdx.y;
  if (it >= A.nitems || param >= A.nparams) {
    return;
  }
  const TmxItem item = A.items[it];
  const TmxSlot sl = A.slots[item.slot];
  const TmxGrain Gr = A.grains[sl.grain];
  const int N = sl.nmax;
  const int ng = sl.ngauss;
  const int m = item.m;
  const ClassDesc D = describe<TR>(N, m, item.cls);
  const int nb = D.nb;
  // (shared memory is sized for classes of at most max_nb members)
  if (nb <= 0 || nb > TMX_MAX_NB || nb > A.max_nb) {
    return;
  }
  const double *T = A.tab + sl.tab;
  const double *S = A.nsc + sl.nsc;
  const double *Wg = A.wig + A.wig_off[sl.wig_n] + (int64_t)m * ng * N * 2;
  const double k2 = Gr.k * Gr.k;
  const cplx k2mr = mkc(Gr.mr * k2, Gr.mi * k2);
  cplx *dQ = A.scratch + param * A.scratch_stride + item.scratch;
  cplx *dR = dQ + (int64_t)nb * nb;
  __shared__ double an_tab[TMX_MAX_NB];
  for (int a = threadIdx.x; a < nb; a += blockDim.x) {
    int ia, na;
    member(D, a, ia, na);
    an_tab[a] = a_n(na);
  }

  // ---------------------------------------------------- tangent assembly
  AsmLayout L;
  L.G = A.chunk_nodes;
  L.NRp = D.NRp;
  L.CT = (nb + TC - 1) / TC;
  L.ncol = L.CT * TC;
  L.ngroups = (D.R1 > 0 && m > 0) ? 2 : 1;
  const int RT = D.NRp / TR;
  cplx *Fs = reinterpret_cast<cplx *>(tmx_tsmem);
  cplx *Ws = Fs + (int64_t)8 * L.G * L.NRp;
  const int ntiles = RT * L.CT;
  const int tstep = (m == 0) ? 2 : 1;
  const int t0 = (m == 0) ? 1 : 0;
  const int per_node = (param == P_M) ? 4 : 8;
  for (int tile0 = 0; tile0 < ntiles; tile0 += NT) {
    const int tile = tile0 + threadIdx.x;
    const bool active = tile < ntiles;
    const int ct = active ? tile % L.CT : 0;
    const int rt = active ? tile / L.CT : 0;
    const int rg = (rt * TR < D.R0p) ? 0 : 1;
    double aj[TR][TC][2], ay[TR][TC][2];
#pragma unroll
    for (int r = 0; r < TR; ++r) {
#pragma unroll
      for (int c = 0; c < TC; ++c) {
        aj[r][c][0] = aj[r][c][1] = ay[r][c][0] = ay[r][c][1] = 0.;
      }
    }
    for (int g0 = 0; g0 < ng; g0 += L.G) {
      __syncthreads();
      build_chunk_tangent(D, L, L.CT * TC, N, m, ng, g0, param, Gr.r_ev, T, S,
                          Wg, k2, k2mr, Fs, Ws, threadIdx.x, blockDim.x, an_tab);
      __syncthreads();
      if (active) {
        const int gmax = min(L.G, ng - g0);
        for (int gl = 0; gl < gmax; ++gl) {
          for (int ts = t0; ts < per_node; ts += tstep) {
            const int kk = 8 * gl + ts;
            const cplx *fr = Fs + (int64_t)kk * L.NRp + rt * TR;
            const cplx *wr = Ws + ((int64_t)rg * 8 * L.G + kk) * L.ncol + ct;
            cplx f[TR], w[TC];
#pragma unroll
            for (int r = 0; r < TR; ++r) {
              f[r] = fr[r];
            }
#pragma unroll
            for (int c = 0; c < TC; ++c) {
              w[c] = wr[c * L.CT];
            }
#pragma unroll
            for (int r = 0; r < TR; ++r) {
#pragma unroll
              for (int c = 0; c < TC; ++c) {
                aj[r][c][0] = fma(f[r].x, w[c].x, aj[r][c][0]);
                aj[r][c][1] = fma(f[r].x, w[c].y, aj[r][c][1]);
                ay[r][c][0] = fma(f[r].y, w[c].x, ay[r][c][0]);
                ay[r][c][1] = fma(f[r].y, w[c].y, ay[r][c][1]);
              }
            }
          }
        }
      }
    }
    if (active) {
#pragma unroll
      for (int r = 0; r < TR; ++r) {
        const int a = padded_member(D, rt * TR + r);
        if (a < 0) {
          continue;
        }
#pragma unroll
        for (int c = 0; c < TC; ++c) {
          const int b = ct + c * L.CT;
          if (b >= nb) {
            continue;
          }
          dQ[(int64_t)a * nb + b] =
              mkc(aj[r][c][0] - ay[r][c][1], aj[r][c][1] + ay[r][c][0]);
          dR[(int64_t)a * nb + b] = mkc(aj[r][c][0], aj[r][c][1]);
        }
      }
    }
  }
  __syncthreads();

  // ---------------------------------------- solve with the saved factors
  const int lda = nb | 1;
  cplx *Am = reinterpret_cast<cplx *>(tmx_tsmem);
  cplx *uinv = Am + (int64_t)nb * lda;
  int *perm = reinterpret_cast<int *>(uinv + nb);
  size_t used = ((size_t)nb * lda + nb) * sizeof(cplx) + nb * sizeof(int);
  used = (used + 15) & ~(size_t)15;
  cplx *X = reinterpret_cast<cplx *>(tmx_tsmem + used);
  int Rchunk = (int)((smem_bytes - used) / (sizeof(cplx) * lda));
  if (Rchunk > nb) {
    Rchunk = nb;
  }
  const cplx *Ls = A.lu + item.scratch;
  const int *ps = reinterpret_cast<const int *>(Ls + (int64_t)nb * nb);
  for (int u = threadIdx.x; u < nb * nb; u += blockDim.x) {
    Am[(u / nb) * lda + (u % nb)] = Ls[u];
  }
  for (int j = threadIdx.x; j < nb; j += blockDim.x) {
    perm[j] = ps[j];
    uinv[j] = cinv(Ls[(int64_t)j * nb + j]);
  }
  __syncthreads();
  const cplx *Tb = A.T + sl.tout + block_offset(N, m);
  cplx *dTb = A.dT + param * A.dT_stride + sl.tout + block_offset(N, m);
  const int w2 = 2 * D.nbb;
  for (int r0 = 0; r0 < nb; r0 += Rchunk) {
    const int R = min(Rchunk, nb - r0);
    // X = -(dRgQ + T_c dQ) for rows r0 .. r0 + R
    for (int u = threadIdx.x; u < R * nb; u += blockDim.x) {
      const int r = u / nb;
      const int b = u % nb;
      const int a = r0 + r;
      int ia, na;
      member(D, a, ia, na);
      const cplx *trow = Tb + (int64_t)(ia * D.nbb + (na - D.nmin)) * w2;
      cplx acc = dR[(int64_t)a * nb + b];
      for (int k = 0; k < nb; ++k) {
        int ik, nk;
        member(D, k, ik, nk);
        acc = cadd(acc, cmul(trow[ik * D.nbb + (nk - D.nmin)], dQ[(int64_t)k * nb + b]));
      }
      X[r * lda + b] = mkc(-acc.x, -acc.y);
    }
    __syncthreads();
    for (int j = 0; j < nb; ++j) {
      for (int r = threadIdx.x; r < R; r += blockDim.x) {
        X[r * lda + j] = cmul(X[r * lda + j], uinv[j]);
      }
      __syncthreads();
      const int rem = nb - j - 1;
      for (int u = threadIdx.x; u < R * rem; u += blockDim.x) {
        const int r = u / rem;
        const int k = j + 1 + u % rem;
        X[r * lda + k] = csub(X[r * lda + k], cmul(X[r * lda + j], Am[j * lda + k]));
      }
      __syncthreads();
    }
    for (int j = nb - 1; j >= 1; --j) {
      for (int u = threadIdx.x; u < R * j; u += blockDim.x) {
        const int r = u / j;
        const int k = u % j;
        X[r * lda + k] = csub(X[r * lda + k], cmul(X[r * lda + j], Am[j * lda + k]));
      }
      __syncthreads();
    }
    for (int u = threadIdx.x; u < R * nb; u += blockDim.x) {
      const int r = u / nb;
      const int b = u % nb;
      const int a = r0 + r;
      int ia, na, ib, nbn;
      member(D, a, ia, na);
      member(D, b, ib, nbn);
      dTb[(int64_t)(ia * D.nbb + (na - D.nmin)) * w2 + ib * D.nbb + (nbn - D.nmin)] =
          X[r * lda + perm[b]];
    }
    __syncthreads();
  }
}

// -------------------------------------- all three parameters of an item --
//
// Classes of at most 32 members. With U = z dF/dz, V = z dW/dw (w = m z the
// argument of the B side; every weight kept) and L = (d ln r^2 / dd) / 2:
//   dW/dm = V + W'/m (W': the terms whose factor is m k^2, which are t = 0, 1
//   for rows of block index 0 and t = 2, 3 for those of 1),
//   dF/dR = U / R, dW/dR = (m / R) V,
//   dF/dd = L U + e_F, dW/dd = L (m V + 2 W) + e_W (e: the d(r'/r)/dd terms).
// So with V' = V + W'/m and U' = U - F' (F': F at the terms of W'),
//   dQ/dm = sum F V' = A,  dQ/dR = (m A + B) / R with B = sum U' W,
//   dQ/dd = sum F (L (m V' + 2 W) + e_W) + (L U' + e_F) W:
// four products of four terms per node instead of the twenty terms of three
// passes, and one build of F, U, W and V instead of three. The products run on
// the FP64 tensor pipe, one 8 x 8 tile (three accumulator sets) per warp, one
// item per CTA; rows are padded per row group, padding is neither cleared nor
// written out. Then x = -(dRgQ + T_c dQ) and both triangular solves with the
// saved factors, C lanes per (parameter, row). dQ/dR leaves out 2 Q / R of the
// weights' R^2 and dRgQ the same of RgQ: they cancel in dRgQ + T dQ.
// Bound by the FP64 pipe (about 2/3 products, 1/3 build) and by the barriers
// of the chunks; 1024 grains of orders 4 to 20, four rounds: classes of at
// most 8 0.70 ms (a warp per item and parameter, entries in registers: 1.67),
// 9..16 0.92 ms (1.90), 17..32 0.73 ms (128 threads per item and parameter:
// 1.58). Measured and not taken: 3 nodes per chunk for more CTAs per SM (0.79
// and 0.96 ms), 4 lanes per row for classes of at most 8 (0.96 ms).
// NC: largest class; NR: its padded rows; WG: nodes per chunk.
template <int NC, int NR, int NTH, int WG>
struct TangentTile {
  static constexpr int LA = NR + 2, LB = NC + 2; // (bank-conflict-free fragments)
  static constexpr int ROW = 10;                 // staged row: Bessel 8, Wigner 2
  static constexpr int A_ELEMS = 12 * WG * LA, B_ELEMS = 24 * WG * LB;
  static constexpr int STAGE = WG * (NC * ROW + TMX_NS); // doubles
  static constexpr int LD = NC + 1, MAT = NC * LD;
  static constexpr size_t CHUNK_BYTES =
      (size_t)(A_ELEMS + B_ELEMS) * sizeof(cplx) + STAGE * sizeof(double);
  static constexpr size_t SOLVE_BYTES = (size_t)7 * MAT * sizeof(cplx);
  static constexpr size_t BYTES = CHUNK_BYTES > SOLVE_BYTES ? CHUNK_BYTES : SOLVE_BYTES;
};

__device__ __forceinline__ void tdmma(double *d, double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, "
      "{%0, %1};\n"
      : "+d"(d[0]), "+d"(d[1])
      : "d"(a), "d"(b));
}

template <int NC, int NR, int NTH, int WG, int C, int MINB>
__global__ void __launch_bounds__(NTH, MINB) k_tangent_tile(TmxTangentArgs A) {
  using Z = TangentTile<NC, NR, NTH, WG>;
  constexpr int LA = Z::LA, LB = Z::LB, LD = Z::LD, ROW = Z::ROW;
  constexpr int NT = NC / C;
  static_assert(NR / 8 * (NC / 8) <= NTH / 32 && 3 * NC <= NTH / C, "thread layout");
  __shared__ double an_s[NC];
  __shared__ cplx uinv[NC];
  __shared__ int at[NC]; // class member of a solved column
  cplx *As = reinterpret_cast<cplx *>(tmx_tsmem); // [F, U', Ud][WG][4][LA]
  cplx *Bs = As + Z::A_ELEMS;                     // [group][V', W, Wd][WG][4][LB]
  double *stg = reinterpret_cast<double *>(Bs + Z::B_ELEMS);
  double *stgS = stg + WG * NC * ROW;
  cplx *dQ = As;              // (after the assembly) [3][NC][LD]
  cplx *dR = dQ + 3 * Z::MAT; // [3][NC][LD]
  cplx *Tc = dR + 3 * Z::MAT; // [NC][LD]
  cplx *LU = dQ;              // (after x)
  const int tid = threadIdx.x;
  const int lane = tid & 31;
  const int warp = tid >> 5;
  const int q = lane & 3;
  const int rr = lane >> 2;
  const TmxItem item = A.items[blockIdx.x];
  const TmxSlot sl = A.slots[item.slot];
  const int N = sl.nmax;
  const int ng = sl.ngauss;
  const int m = item.m;
  const ClassDesc D = describe<8>(N, m, item.cls);
  const int nb = D.nb;
  if (nb <= 0 || nb > NC || D.NRp > NR) {
    return;
  }
  const TmxGrain Gr = A.grains[sl.grain];
  const double *T = A.tab + sl.tab;
  const double *S = A.nsc + sl.nsc;
  const double *Wg = A.wig + A.wig_off[sl.wig_n] + (int64_t)m * ng * N * 2;
  const double k2 = Gr.k * Gr.k;
  const cplx mc = mkc(Gr.mr, Gr.mi);
  const cplx minv = cinv_lu(mc);
  const cplx k2mr = mkc(Gr.mr * k2, Gr.mi * k2);
  const int ngroups = (D.R1 > 0 && m > 0) ? 2 : 1;
  const auto stage = [&](int g0) {
    const int live = min(WG, ng - g0);
    for (int u = tid; u < live * nb * 5; u += NTH) {
      const int gl = u / (nb * 5);
      const int v = u - gl * nb * 5;
      const int a = v / 5, p = v - 5 * a;
      int ia, n;
      member(D, a, ia, n);
      const int64_t o = (int64_t)(g0 + gl) * N + (n - 1);
      const double *src = (p < 4) ? T + o * TMX_NQ + 2 * p : Wg + o * 2;
      const unsigned dst =
          (unsigned)__cvta_generic_to_shared(stg + (gl * NC + a) * ROW + 2 * p);
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(src)
                   : "memory");
    }
    for (int u = tid; u < live * (TMX_NS / 2); u += NTH) {
      const unsigned dst = (unsigned)__cvta_generic_to_shared(stgS + 2 * u);
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst),
                   "l"(S + (int64_t)g0 * TMX_NS + 2 * u)
                   : "memory");
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
  stage(0);
  if (tid < nb) {
    int ia, n;
    member(D, tid, ia, n);
    an_s[tid] = a_n(n);
  }
  // this warp's tile
  const int nct = (nb + 7) >> 3;
  const int trow = (warp / nct) * 8, tcol = (warp % nct) * 8;
  const bool tile = trow < D.NRp;
  const cplx *fr = As + q * LA + trow + rr;
  const cplx *wr = Bs + (trow < D.R0p ? 0 : Z::B_ELEMS / 2) + q * LB + tcol + rr;
  double aA[4][2], aB[4][2], aD[4][2]; // (j re, j im, y re, y im)
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    aA[e][0] = aA[e][1] = aB[e][0] = aB[e][1] = aD[e][0] = aD[e][1] = 0.;
  }
  for (int g0 = 0; g0 < ng; g0 += WG) {
    asm volatile("cp.async.wait_all;\n" ::: "memory");
    __syncthreads(); // the chunk's rows are there; the fragments are free
    const int live = min(WG, ng - g0);
    const int nunit = live * nb;
    for (int u = tid; u < nunit * (1 + ngroups); u += NTH) {
      const int side = u / nunit; // 0: A side, 1, 2: B side of group 0, 1
      const int v = u - side * nunit;
      const int gl = v / nb;
      const int a = v - gl * nb;
      int ib, n;
      member(D, a, ib, n);
      const double *r = stg + (gl * NC + a) * ROW;
      const double *s = stgS + gl * TMX_NS;
      const double d = r[8], dd = r[9];
      const double nn = n * (n + 1.);
      const double z = s[TMX_NS_KR];
      const double drr = s[TMX_NS_DRR], ddrr = s[TMX_NS_DDRR_DD];
      const double L = 0.5 * s[TMX_NS_DLNR2_DD];
      if (side == 0) {
        const double iz = s[TMX_NS_KRINV];
        const int row = (a < D.R0) ? a : D.R0p + a - D.R0;
        cplx *o = As + gl * 4 * LA + row;
        const double qd = nn * drr * d, qe = nn * ddrr * d * iz;
        double F[2][4], U[2][4], E[2];
#pragma unroll
        for (int y = 0; y < 2; ++y) {
          const double h = r[2 * y], dh = r[2 * y + 1];
          const double hi = h * iz;
          const double zh = z * dh - h;            // z h'
          const double zdh = nn * hi - z * h - dh; // z (dh)'
          F[y][0] = d * h;
          F[y][1] = dd * h;
          F[y][2] = d * dh;
          F[y][3] = dd * dh + qd * hi;
          U[y][0] = d * zh;
          U[y][1] = dd * zh;
          U[y][2] = d * zdh;
          U[y][3] = dd * zdh + qd * (dh - 2. * hi);
          E[y] = qe * h;
        }
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          const bool mr = (t < 2) == (ib == 0);
          const cplx f = mkc(F[0][t], F[1][t]);
          const cplx g = mr ? mkc(U[0][t] - f.x, U[1][t] - f.y) : mkc(U[0][t], U[1][t]);
          o[t * LA] = f;
          o[(4 * WG + t) * LA] = g;
          o[(8 * WG + t) * LA] = (t == 3) ? mkc(L * g.x + E[0], L * g.y + E[1])
                                          : mkc(L * g.x, L * g.y);
        }
        continue;
      }
      const int ia = (side == 1) ? D.iA : D.iB;
      const bool dg = ia == ib;
      const cplx jm = mkc(r[4], r[5]), djm = mkc(r[6], r[7]);
      const cplx iw = mkc(s[TMX_NS_KRMRINV_RE], s[TMX_NS_KRMRINV_IM]);
      const cplx jw = cmul(jm, iw), djw = cmul(djm, iw), jw2 = cmul(jw, iw);
      const cplx jp = csub(djm, jw);                           // j'
      const cplx djp = csub(csub(cscale(jw2, nn), jm), djw);   // (dj)'
      const cplx jwp = csub(djw, cscale(jw2, 2.));             // (j / w)'
      const double qd = nn * drr * d;
      const double wr2 = s[TMX_NS_W] * s[TMX_NS_R2];
      const double beta = s[TMX_NS_SININV] * m * wr2;
      const double wm = (double)(m * m) * s[TMX_NS_SIN2INV] * wr2;
      const cplx c1 = (ia == 0) ? k2mr : mkc(k2, 0.);
      const cplx c2 = (ia == 0) ? mkc(k2, 0.) : k2mr;
      const cplx ch = dg ? c1 : mkc(-c1.y * beta, c1.x * beta);
      const cplx cl = dg ? mkc(-c2.x, -c2.y) : mkc(-c2.y * beta, c2.x * beta);
      // weights of the terms' G (in the order of the terms)
      const double w0 = dg ? wm : 1., w1 = dg ? wr2 : 1.;
      const cplx G1 = cscale(djm, d), G2 = cadd(cscale(djm, dd), cscale(jw, qd));
      const cplx G3 = cscale(jm, d), G4 = cscale(jm, dd);
      const cplx P1 = cscale(djp, z * d);
      const cplx P2 = cadd(cscale(djp, z * dd), cscale(jwp, z * qd));
      const cplx P3 = cscale(jp, z * d), P4 = cscale(jp, z * dd);
      const cplx ex = cscale(jw, nn * d * ddrr); // of G2
      cplx *o = Bs + (side == 1 ? 0 : Z::B_ELEMS / 2) + gl * 4 * LB + a;
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const cplx g = dg ? (t == 0 ? G1 : t == 1 ? G2 : t == 2 ? G3 : G4)
                          : (t == 0 ? G4 : t == 1 ? G3 : t == 2 ? G2 : G1);
        const cplx pv = dg ? (t == 0 ? P1 : t == 1 ? P2 : t == 2 ? P3 : P4)
                           : (t == 0 ? P4 : t == 1 ? P3 : t == 2 ? P2 : P1);
        const cplx cw = cscale((t < 2) ? ch : cl, (t & 1) ? w1 : w0);
        const cplx W = cmul(cw, g);
        cplx V = cmul(cw, pv);
        if ((t < 2) == (ia == 0)) {
          V = cadd(V, cmul(W, minv));
        }
        const cplx mv = cmul(mc, V);
        cplx X = mkc(L * (mv.x + 2. * W.x), L * (mv.y + 2. * W.y));
        if (dg ? t == 1 : t == 2) {
          X = cadd(X, cmul(cw, ex));
        }
        o[t * LB] = V;
        o[(4 * WG + t) * LB] = W;
        o[(8 * WG + t) * LB] = X;
      }
    }
    __syncthreads();
    if (g0 + WG < ng) {
      stage(g0 + WG);
    }
    if (tile) {
      for (int gl = 0; gl < live; ++gl) {
        const cplx f = fr[gl * 4 * LA], u = fr[(4 * WG + gl * 4) * LA],
                   e = fr[(8 * WG + gl * 4) * LA];
        const cplx v = wr[gl * 4 * LB], w = wr[(4 * WG + gl * 4) * LB],
                   x = wr[(8 * WG + gl * 4) * LB];
        tdmma(aA[0], f.x, v.x);
        tdmma(aA[1], f.x, v.y);
        tdmma(aA[2], f.y, v.x);
        tdmma(aA[3], f.y, v.y);
        tdmma(aB[0], u.x, w.x);
        tdmma(aB[1], u.x, w.y);
        tdmma(aB[2], u.y, w.x);
        tdmma(aB[3], u.y, w.y);
        tdmma(aD[0], f.x, x.x);
        tdmma(aD[1], f.x, x.y);
        tdmma(aD[2], f.y, x.x);
        tdmma(aD[3], f.y, x.y);
        tdmma(aD[0], e.x, w.x);
        tdmma(aD[1], e.x, w.y);
        tdmma(aD[2], e.y, w.x);
        tdmma(aD[3], e.y, w.y);
      }
    }
  }
  __syncthreads();
  // dQ = dG^j + i dG^y, dRgQ = dG^j, by parameter
  const int ra = tile ? padded_member(D, trow + rr) : -1;
  if (ra >= 0) {
    const double ri = 1. / Gr.r_ev;
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int b = tcol + 2 * q + e;
      if (b < nb) {
        const double sc = an_s[ra] * an_s[b];
        const int o = ra * LD + b;
        const cplx Rm = mkc(aA[0][e] * sc, aA[1][e] * sc);
        const cplx Qm = mkc((aA[0][e] - aA[3][e]) * sc, (aA[1][e] + aA[2][e]) * sc);
        const cplx Rb = mkc(aB[0][e] * sc, aB[1][e] * sc);
        const cplx Qb = mkc((aB[0][e] - aB[3][e]) * sc, (aB[1][e] + aB[2][e]) * sc);
        dR[P_M * Z::MAT + o] = Rm;
        dQ[P_M * Z::MAT + o] = Qm;
        dR[P_R * Z::MAT + o] = cscale(cadd(cmul(mc, Rm), Rb), ri);
        dQ[P_R * Z::MAT + o] = cscale(cadd(cmul(mc, Qm), Qb), ri);
        dR[P_D * Z::MAT + o] = mkc(aD[0][e] * sc, aD[1][e] * sc);
        dQ[P_D * Z::MAT + o] =
            mkc((aD[0][e] - aD[3][e]) * sc, (aD[1][e] + aD[2][e]) * sc);
      }
    }
  }
  // T_c (class order) of the forward solve, 1 / U_jj and the column order
  const cplx *Ls = A.lu + item.scratch;
  const int *ps = reinterpret_cast<const int *>(Ls + (int64_t)nb * nb);
  const cplx *Tb = A.T + sl.tout + block_offset(N, m);
  const int w2 = 2 * D.nbb;
  for (int u = tid; u < nb * nb; u += NTH) {
    const int a = u / nb;
    const int k = u - a * nb;
    int ia, na, ik, nk;
    member(D, a, ia, na);
    member(D, k, ik, nk);
    Tc[a * LD + k] =
        Tb[(int64_t)(ia * D.nbb + (na - D.nmin)) * w2 + ik * D.nbb + (nk - D.nmin)];
  }
  for (int j = tid; j < nb; j += NTH) {
    at[ps[j]] = j;
    uinv[j] = cinv_lu(Ls[(int64_t)j * nb + j]);
  }
  __syncthreads();
  // x = -(dRgQ + T_c dQ) of row a of parameter p: columns c + C t in x[t]
  const int c = tid % C;
  const int p = (tid / C) / NC, a = (tid / C) % NC;
  const bool act = p < A.nparams && p < 3 && a < nb;
  cplx x[NT];
#pragma unroll
  for (int t = 0; t < NT; ++t) {
    const int k = c + C * t;
    x[t] = (act && k < nb) ? dR[p * Z::MAT + a * LD + k] : mkc(0., 0.);
  }
  if (act) {
    for (int k = 0; k < nb; ++k) {
      const cplx tk = Tc[a * LD + k];
      const cplx *qk = dQ + p * Z::MAT + k * LD + c;
#pragma unroll
      for (int t = 0; t < NT; ++t) {
        if (c + C * t < nb) {
          const cplx v = qk[C * t];
          x[t].x = fma(tk.x, v.x, fma(-tk.y, v.y, x[t].x));
          x[t].y = fma(tk.x, v.y, fma(tk.y, v.x, x[t].y));
        }
      }
    }
  }
#pragma unroll
  for (int t = 0; t < NT; ++t) {
    x[t] = mkc(-x[t].x, -x[t].y);
  }
  __syncthreads(); // dQ is free
  for (int u = tid; u < nb * nb; u += NTH) {
    LU[(u / nb) * LD + (u % nb)] = Ls[u];
  }
  __syncthreads();
  // X U = x (forward over columns), then Y L = X (backward, L unit lower)
#pragma unroll
  for (int tj = 0; tj < NT; ++tj) {
    if (tj * C < nb) {
      for (int cj = 0; cj < C; ++cj) {
        const int j = tj * C + cj;
        if (j >= nb) {
          break;
        }
        if (c == cj) {
          x[tj] = cmul(x[tj], uinv[j]);
        }
        cplx xj;
        xj.x = __shfl_sync(0xffffffffu, x[tj].x, cj, C);
        xj.y = __shfl_sync(0xffffffffu, x[tj].y, cj, C);
#pragma unroll
        for (int t = tj; t < NT; ++t) {
          const int k = c + C * t;
          if (k > j && k < nb) {
            x[t] = csub(x[t], cmul(xj, LU[j * LD + k]));
          }
        }
      }
    }
  }
#pragma unroll
  for (int tj = NT - 1; tj >= 0; --tj) {
    if (tj * C < nb) {
      for (int cj = min(C, nb - tj * C) - 1; cj >= 0; --cj) {
        const int j = tj * C + cj;
        cplx xj;
        xj.x = __shfl_sync(0xffffffffu, x[tj].x, cj, C);
        xj.y = __shfl_sync(0xffffffffu, x[tj].y, cj, C);
#pragma unroll
        for (int t = 0; t <= tj; ++t) {
          const int k = c + C * t;
          if (k < j) {
            x[t] = csub(x[t], cmul(xj, LU[j * LD + k]));
          }
        }
      }
    }
  }
  if (act) {
    int ia, na;
    member(D, a, ia, na);
    cplx *dTr = A.dT + p * A.dT_stride + sl.tout + block_offset(N, m) +
                (int64_t)(ia * D.nbb + (na - D.nmin)) * w2;
#pragma unroll
    for (int t = 0; t < NT; ++t) {
      const int k = c + C * t;
      if (k < nb) {
        int ib, nbn;
        member(D, at[k], ib, nbn);
        dTr[ib * D.nbb + (nbn - D.nmin)] = x[t];
      }
    }
  }
}

template <int NC, int NR, int NTH, int WG, int C, int MINB>
static void launch_tangent_tile(const TmxTangentArgs &a, cudaStream_t stream) {
  constexpr size_t smem = TangentTile<NC, NR, NTH, WG>::BYTES;
  cudaFuncSetAttribute(k_tangent_tile<NC, NR, NTH, WG, C, MINB>,
                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  k_tangent_tile<NC, NR, NTH, WG, C, MINB><<<a.nitems, NTH, smem, stream>>>(a);
}

size_t tmx_tangent_smem_bytes(int max_nb, int chunk_nodes) {
  const int nrp = (max_nb + 3) / 4 * 4 + 4;
  const int ncol = (max_nb + 3) / 4 * 4;
  const size_t asm_bytes =
      ((size_t)8 * chunk_nodes * nrp + (size_t)2 * 8 * chunk_nodes * ncol) *
      sizeof(cplx);
  const int lda = max_nb | 1;
  size_t lu = ((size_t)max_nb * lda + max_nb) * sizeof(cplx) + max_nb * sizeof(int);
  lu = (lu + 15) & ~(size_t)15;
  const int rows = max_nb < 8 ? max_nb : 8;
  size_t lu_total = lu + (size_t)rows * lda * sizeof(cplx);
  const size_t full = lu + (size_t)max_nb * lda * sizeof(cplx);
  if (full <= 200 * 1024) {
    lu_total = full;
  }
  return asm_bytes > lu_total ? asm_bytes : lu_total;
}

template <int TR, int TC, int NT, int MINB>
static void launch_tangent(const TmxTangentArgs &a, size_t smem,
                           cudaStream_t stream) {
  static int attr_dev = -1;
  int dev = 0;
  cudaGetDevice(&dev);
  if (attr_dev != dev) {
    // the block limit (227 KiB) covers the kernel's static shared memory too
    cudaFuncAttributes fa;
    cudaFuncGetAttributes(&fa, k_tangent<TR, TC, NT, MINB>);
    cudaFuncSetAttribute(k_tangent<TR, TC, NT, MINB>,
                         cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)(227 * 1024 - fa.sharedSizeBytes));
    attr_dev = dev;
  }
  dim3 grid(a.nitems, a.nparams);
  k_tangent<TR, TC, NT, MINB><<<grid, NT, smem, stream>>>(a, smem);
}

void tmx_launch_tangents(const TmxTangentArgs &a, cudaStream_t stream) {
  if (a.nitems <= 0 || a.nparams <= 0) {
    return;
  }
  // One variant per padded size: the tile count sets the warps of a CTA, the
  // class size its shared memory (33, 47 and 118 KB: 6, 4 and 1 CTAs per SM).
  // Above 32 the three parameters' matrices no longer fit (7 nb^2 entries) and
  // each parameter has a CTA of its own.
  if (a.max_nb <= 8) {
    launch_tangent_tile<8, 16, 64, 4, 2, 6>(a, stream);
    return;
  }
  if (a.max_nb <= 16) {
    launch_tangent_tile<16, 16, 128, 4, 2, 4>(a, stream);
    return;
  }
  if (a.max_nb <= 32) {
    launch_tangent_tile<32, 32, 512, 4, 4, 1>(a, stream);
    return;
  }
  launch_tangent<4, 4, 256, 1>(a, tmx_tangent_smem_bytes(a.max_nb, a.chunk_nodes), stream);
}
